// Column passes of the fused FFT: transforms along an outer axis (y or z), the CTA's NV
// vectors being adjacent x positions (see pfb_fft.cuh).  Instantiated in pfb_fft_cols_*.cu.
#pragma once

#include "pfb_fft_passes.cuh"

namespace pfb {
namespace fft {

// element `i` strides of `bytes` bytes from p (one multiply-add for the address)
template <class E>
__device__ __forceinline__ E *step(E *p, int i, int bytes) {
    return reinterpret_cast<E *>(reinterpret_cast<uintptr_t>(p) + (int64_t)i * bytes);
}
// i mod n for 0 <= i < 2 n
__device__ __forceinline__ int wrap(int i, int n) { return (int)min((unsigned)i, (unsigned)(i - n)); }

// reads position p of a column: source row (p + hn) mod n of a forward pass (the
// fftshift rotation; rows past the input extent are the zero padding), row p of an
// inverse one
template <bool FWD>
struct ColLoad {
    const float2 *src;
    int bytes, n, hn, lin;  // bytes: stride along the axis
    __device__ __forceinline__ float2 operator()(int p) const {
        // plain loads: a pass may run in place (a CTA reads its columns before it writes)
        if (!FWD) return *step(src, p, bytes);
        const int i = wrap(p + hn, n);
        return i < lin ? *step(src, i, bytes) : make_float2(0.f, 0.f);
    }
};

// the same of a forward first pass: times the B0 factor of the plane's segment (CL), the
// deapodisation and the scale.  Without a branch around the loads, so that those of a
// butterfly are in flight together
template <bool CL>
struct ColLoadImage {
    const float2 *src;
    int bytes, n, hn, lin;
    const float *apod;  // null: no deapodisation
    const float2 *cl;
    float a;
    __device__ __forceinline__ float2 operator()(int p) const {
        const int i = wrap(p + hn, n);
        const bool in = i < lin;
        float2 v = in ? __ldg(step(src, i, bytes)) : make_float2(0.f, 0.f);
        if (CL) v = cmul(v, in ? __ldg(step(cl, i, bytes)) : make_float2(0.f, 0.f));
        const float f = apod ? a * __ldg(apod + (in ? i : 0)) : a;
        return make_float2(v.x * f, v.y * f);
    }
};

// writes result k of a column: row k of a forward pass; of an inverse pass the row whose
// inverse-transform position is (n - k) mod n, cropped to lout rows
template <bool FWD>
struct ColStore {
    float2 *dst;
    int bytes, n, hn, lout;
    bool on;
    __device__ __forceinline__ void operator()(int k, float2 v) const {
        const int o = FWD ? k : wrap(wrap(n - k, n) + hn, n);
        if ((FWD || o < lout) && on) *step(dst, o, bytes) = v;
    }
};

// the last pass of an adjoint: the transform times the deapodisation and the scale, with
// SEG the sum over the B0 segments of conj(C_l) times their transforms (partial sums in
// shared memory: a position is always the same thread's), and the optional accumulation
template <bool SEG>
struct ColStoreImage {
    float2 *dst;
    int bytes, n, hn, lout;
    bool on;
    const float *apod;  // null: no deapodisation
    float a;
    bool accumulate;
    const float2 *cl;   // SEG: the segment's factors
    float2 *acc;        // this column's partial sums, pitch `pitch`
    int pitch;
    bool first, last;
    __device__ __forceinline__ void operator()(int k, float2 v) const {
        const int o = wrap(wrap(n - k, n) + hn, n);
        const bool in = o < lout && on;
        // the factors first and without a branch, so that those of a butterfly are in flight
        // together
        const int oc = o < lout ? o : 0;
        const float f = apod ? a * __ldg(apod + oc) : a;
        if (SEG) v = cmulc(v, __ldg(step(cl, oc, bytes)));
        if (!in) return;
        if (SEG) {
            if (!first) v = cadd(v, acc[o * pitch]);
            if (!last) {
                acc[o * pitch] = v;
                return;
            }
        }
        v = make_float2(v.x * f, v.y * f);
        float2 *d = step(dst, o, bytes);
        if (accumulate) v = cadd(v, *d);
        *d = v;
    }
};

// A CTA: NV adjacent columns of one (plane, mid).  What bounds it in 3D is HBM: 200^3, 32
// coils, z pass 1.05 ms (4.4 TB/s, 67 % of the copy rate), y pass 1.11 ms (5.2 TB/s, 79 %);
// 128^3 in 128 points 5.4 to 6.4 TB/s.  Groups of radices above 16 run at half the warps (128
// registers): 512 points, 256 images of 256^2, 96 us (3.6 TB/s).
template <int MODE, int NV, int G>
__global__ void __launch_bounds__(kMaxThreads, min_blocks(big_group(G))) col_kernel(const ColPass P) {
    extern __shared__ __align__(16) float2 fsm[];
    using A = ColAddr<NV>;
    const int n = P.fa.n, T = P.T;
    const int v = threadIdx.x % NV, stream = threadIdx.x / NV;
    const A ad{v};
    float2 *b0 = fsm, *b1 = fsm + (P.fa.nst > 2 ? A::size(n) : 0);
    int xc, mid;
    const int plane = P.dmid.split(P.dx.split(blockIdx.x, xc), mid);
    const int x = xc * NV + v;
    const bool xin = x < P.X;
    const int xs = xin ? x : P.X - 1;  // in-bounds address for columns past the edge
    const int hn = P.nax / 2;
    const int Kc = P.ch.K ? P.ch.K : 1;
    float a = P.factor;
    if (MODE == kImageIn || MODE == kImageOut) {
        if (P.apod_mid) a *= __ldg(P.apod_mid + mid);
        if (P.apod_x) a *= __ldg(P.apod_x + xs);
    }
    if constexpr (MODE == kImageIn) {  // grid plane (grp, chn) <- image plane (b, c), segment l
        int chn, k, b;
        const int grp = P.dnch.split(plane, chn), lb = P.dk.split(chn, k), l = P.db.split(lb, b);
        const int c = P.ch.K ? k : grp;
        const int64_t off = (int64_t)mid * P.in_mid + xs;
        const float2 *src = P.src + ((int64_t)b * P.C + c) * P.nvol + off;
        ColStore<true> st{P.dst + (int64_t)plane * P.out_plane + (int64_t)mid * P.out_mid + x, (int)P.out_ax * 8, n, hn, n,
                          xin};
        if (P.Cl) {
            ColLoadImage<true> ld{src, (int)P.in_ax * 8, n, hn, P.lin, P.apod_ax, P.Cl + (int64_t)l * P.nvol + off, a};
            run<G>(P.fa, stream, T, ad, b0, b1, ld, st);
        } else {
            ColLoadImage<false> ld{src, (int)P.in_ax * 8, n, hn, P.lin, P.apod_ax, nullptr, a};
            run<G>(P.fa, stream, T, ad, b0, b1, ld, st);
        }
    } else if constexpr (MODE == kForward || MODE == kInverse) {
        constexpr bool F = MODE == kForward;
        ColLoad<F> ld{P.src + (int64_t)plane * P.in_plane + (int64_t)mid * P.in_mid + xs, (int)P.in_ax * 8, n, hn, P.lin};
        ColStore<F> st{P.dst + (int64_t)plane * P.out_plane + (int64_t)mid * P.out_mid + x, (int)P.out_ax * 8, n, hn,
                       P.lout, xin};
        run<G>(P.fa, stream, T, ad, b0, b1, ld, st);
    } else {  // image plane (b, c) <- grid planes of its segments
        int c;
        const int b = P.dc.split(plane, c);
        const int grp = P.ch.K ? 0 : c;
        const int64_t off = (int64_t)mid * P.out_mid;
        float2 *dst = P.dst + (int64_t)plane * P.nvol + off + x;
        const float2 *src = P.src + (int64_t)grp * P.ch.nch * P.in_plane + (int64_t)mid * P.in_mid + xs;
        auto chan = [&](int l) { return P.ch.K ? (l * P.ch.B + b) * Kc + c : l * P.ch.B + b; };
        if (!P.Cl) {  // one segment
            ColLoad<false> ld{src + chan(0) * P.in_plane, (int)P.in_ax * 8, n, hn, P.lin};
            ColStoreImage<false> st{dst, (int)P.out_ax * 8, n, hn, P.lout, xin, P.apod_ax, a, P.accumulate != 0};
            run<G>(P.fa, stream, T, ad, b0, b1, ld, st);
            return;
        }
        float2 *acc = fsm + (P.fa.nst > 2 ? 2 : 1) * A::size(n) + v;
        for (int l = 0; l < P.ch.L; ++l) {
            ColLoad<false> ld{src + chan(l) * P.in_plane, (int)P.in_ax * 8, n, hn, P.lin};
            ColStoreImage<true> st{dst, (int)P.out_ax * 8, n, hn, P.lout, xin, P.apod_ax, a, P.accumulate != 0,
                                   P.Cl + (int64_t)l * P.nvol + off + xs, acc, NV, l == 0,
                                   l + 1 == P.ch.L};
            if (l > 0) __syncthreads();  // the previous segment's last stage has read its buffer
            run<G>(P.fa, stream, T, ad, b0, b1, ld, st);
        }
    }
}

template <int MODE, int NV, int G>
int launch_nv(ColPass P, cudaStream_t s) {
    const int64_t blocks = (int64_t)P.nplanes * P.nmid * ((P.X + NV - 1) / NV);
    if (blocks >= (1LL << 31)) return fail(PFB_ERR_UNSUPPORTED, "too many vectors for the fused FFT");
    const int bufs = (P.fa.nst > 2 ? 2 : 1) + (MODE == kImageOut && P.Cl ? 1 : 0);
    const size_t smem = (size_t)bufs * ColAddr<NV>::size(P.fa.n) * sizeof(float2);
    P.T = streams(P.fa, NV, smem, blocks);
    P.dx = Div((P.X + NV - 1) / NV);
    P.dmid = Div(P.nmid);
    P.dnch = Div(P.ch.nch);
    P.dk = Div(P.ch.K);
    P.db = Div(P.ch.B);
    P.dc = Div(P.C);
    auto k = col_kernel<MODE, NV, G>;
    PFB_RAISE_SMEM(k, (int)smem);
    k<<<(unsigned)blocks, NV * P.T, smem, s>>>(P);
    PFB_CHECK_LAUNCH();
    return PFB_OK;
}

template <int MODE, int G>
int launch_col_mode(const ColPass &P, cudaStream_t s) {
    const int64_t tiles = (int64_t)P.nplanes * P.nmid * ((P.X + 15) / 16);
    if constexpr (big_group(G)) return launch_nv<MODE, 8, G>(P, s);
    else return narrow_tiles(P.fa.n, tiles) ? launch_nv<MODE, 8, G>(P, s) : launch_nv<MODE, 16, G>(P, s);
}

}  // namespace fft
}  // namespace pfb
