// The Gram operator's middle pass: forward transform along x, the per-voxel product with
// the Gram kernel, inverse transform along x, in one read and one write of the grid rows
// (src/pyfourier/_sparsegram/_sparsegram.py:56-81 runs FFT, product and inverse FFT one
// after the other; out[v] = T[v] @ in[v] is the evident intent of _bmatvec/_bdot.py:16-115).
//
// The embedding's shift does not change a product with a function of frequency, so the
// image sits at the grid's origin: the outer axes' passes (pfb_fft_cols.cuh) and this one
// read N rows and zero-pad them, and write back N rows; no grid of the full size exists
// and pad, crop and product cost no pass of their own.  A CTA holds V vectors of one grid
// row: all K planes of `nbv` batch items (or, for the elementwise kernel, V batch items of
// one plane), so that a kernel row T is read once per CTA.  Instantiated in
// pfb_fft_gram.cu and pfb_fft_gram_big.cu.
#pragma once

#include "pfb_fft_passes.cuh"

namespace pfb {
namespace fft {

// Elementwise kernel, two stages R0 x R1: forward, product and inverse of the thread's
// vector, ld(position) and st(position) as in run.  A thread's results of the last forward
// stage, frequencies i + k R0, are its points of a first stage of radix R1: they are
// multiplied in registers and the inverse runs the radices in the other order.  The row is
// in shared memory twice instead of five times (256 points, 8 images of 128^3:
// 520 -> 440 us).
template <int R0, int R1, class L, class S>
__device__ __forceinline__ void gram_two(const float2 *__restrict__ tw, const float2 *__restrict__ sw,
                                         const float2 *__restrict__ kern, int stream, int T, RowAddr ad, float2 *b0,
                                         float2 *b1, L &ld, S &st) {
    constexpr int S0 = RowAddr::between(R0), S1 = RowAddr::between(R1);
    for (int i = stream; i < R1; i += T) {
        float2 a[R0];
#pragma unroll
        for (int q = 0; q < R0; ++q) a[q] = ld(i + q * R1);
        dft<R0>(a);
        float2 *d = b0 + ad.at(i * S0);
#pragma unroll
        for (int k = 0; k < R0; ++k) d[k] = a[k];
    }
    __syncthreads();
    for (int i = stream; i < R0; i += T) {
        float2 a[R1];
#pragma unroll
        for (int q = 0; q < R1; ++q) a[q] = b0[ad.at(i + q * S0)];
        twiddle<R1>(a, tw, R0, i);
        dft<R1>(a);
#pragma unroll
        for (int k = 0; k < R1; ++k) a[k] = cmul(__ldg(kern + i + k * R0), a[k]);
        dft<R1>(a);
        float2 *d = b1 + ad.at(i * S1);
#pragma unroll
        for (int k = 0; k < R1; ++k) d[k] = a[k];
    }
    __syncthreads();
    for (int i = stream; i < R1; i += T) {
        float2 a[R0];
#pragma unroll
        for (int q = 0; q < R0; ++q) a[q] = b1[ad.at(i + q * S1)];
        twiddle<R0>(a, sw, R1, i);
        dft<R0>(a);
#pragma unroll
        for (int k = 0; k < R0; ++k) st(i + k * R1, a[k]);
    }
}

// float2 of shared memory between vectors: as the row passes, and the rows of gram_two
inline __host__ __device__ int gram_pitch(const FftAxis &fa) {
    const int two = fa.nst == 2 ? fa.radix[0] * RowAddr::between(fa.radix[1]) | 1 : 0;
    return two > RowAddr::pitch(fa.n) ? two : RowAddr::pitch(fa.n);
}

template <bool LOWRANK, int G>
__global__ void __launch_bounds__(kMaxThreads, min_blocks(big_group(G))) gram_rows_kernel(const GramRows P) {
    extern __shared__ __align__(16) float2 fsm[];
    const int n = P.fa.n, T = P.T, N0 = P.N0, K = P.K;
    const int pitch = LOWRANK ? RowAddr::pitch(n) : gram_pitch(P.fa);
    int stream;
    const int v = P.dt.split(threadIdx.x, stream);
    const RowAddr ad{v * pitch};
    // blocks: batch groups fastest (they share the kernel row), then planes of the
    // elementwise kernel, rows, segments
    int bg, c = 0, row, k;
    int blk = P.dbg.split(blockIdx.x, bg);
    if (!LOWRANK) blk = P.dk.split(blk, c);
    const int l = P.drow.split(blk, row);
    const int b0i = bg * P.nbv, nbc = min(P.nbv, P.batch - b0i);
    // vector v: batch item b0i + bi, plane k
    int bi = v;
    if (LOWRANK) bi = P.dk.split(v, k);
    else k = c;
    const bool on = bi < nbc;
    const int64_t plane = ((int64_t)l * P.batch + b0i + (on ? bi : 0)) * K + k;
    float2 *g = P.grid + (plane * P.rows + row) * N0;
    float2 *B0 = fsm, *B1 = fsm + P.V * pitch;
    auto ld = [&](int p) { return p < N0 ? g[p] : make_float2(0.f, 0.f); };
    auto st = [&](int q, float2 r) {
        const int o = (int)min((unsigned)(n - q), 0u - (unsigned)q);  // (n - q) mod n
        if (on && o < N0) g[o] = r;
    };
    if (!LOWRANK && P.fa.nst == 2) {
        const float2 *tr = P.kern + ((int64_t)l * K + c) * P.gvol + (int64_t)row * n;
        switch (P.fa.radix[0] * 32 + P.fa.radix[1]) {
#define X(R0, R1) \
    case R0 * 32 + R1: \
        if constexpr (!LOWRANK && group_of(R0) == G) \
            gram_two<R0, R1>(P.fa.tw + P.fa.twoff[1], P.fa.tw + P.fa.swapoff, tr, stream, T, ad, B0, B1, ld, st); \
        return;
            PFB_FFT_TWO(X) PFB_FFT_TWO_BIG(X)
#undef X
            default: break;
        }
    }
    float2 *M = P.fa.nst % 2 == 0 ? B1 : B0;  // the buffer that the last stage does not read
    auto sm = [&](int q, float2 r) { M[ad.at(q)] = r; };
    run<G>(P.fa, stream, T, ad, B0, B1, ld, sm);
    __syncthreads();
    float2 *O = M == B1 ? B0 : B1;
    if constexpr (!LOWRANK) {
        const float2 *tr = P.kern + ((int64_t)l * K + c) * P.gvol + (int64_t)row * n;
        for (int x = threadIdx.x; x < n; x += blockDim.x) {
            const float2 t = __ldg(tr + x);
            float2 *m = M + x;
            for (int b = 0; b < nbc; ++b) m[b * pitch] = cmul(t, m[b * pitch]);
        }
        O = M;
    } else {
        // thread (x, i): output plane i of point x of every batch item, into the other
        // buffer; consecutive threads read consecutive rows of the K x K matrices
        const float2 *tr = P.kern + ((int64_t)l * P.gvol + (int64_t)row * n) * (K * K);
        for (int e = threadIdx.x; e < n * K; e += blockDim.x) {
            int i;
            const int x = P.dk.split(e, i);
            const float2 *te = tr + (int64_t)e * K;
            float2 t[8];
            if (K == 4) {  // 32-byte rows
                const float4 u = __ldg(reinterpret_cast<const float4 *>(te)), w = __ldg(reinterpret_cast<const float4 *>(te) + 1);
                t[0] = make_float2(u.x, u.y);
                t[1] = make_float2(u.z, u.w);
                t[2] = make_float2(w.x, w.y);
                t[3] = make_float2(w.z, w.w);
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) t[j] = j < K ? __ldg(te + j) : make_float2(0.f, 0.f);
            }
            const float2 *m = M + x;
            float2 *o = O + i * pitch + x;
            for (int b = 0; b < nbc; ++b, m += K * pitch, o += K * pitch) {
                float2 acc = cmul(t[0], m[0]);
#pragma unroll
                for (int j = 1; j < 8; ++j) {
                    if (j >= K) break;
                    const float2 q = cmul(t[j], m[j * pitch]);
                    acc.x += q.x;
                    acc.y += q.y;
                }
                *o = acc;
            }
        }
    }
    __syncthreads();
    // inverse: the forward transform read reversed
    auto lm = [&](int p) { return O[ad.at(p)]; };
    run<G>(P.fa, stream, T, ad, O == B1 ? B0 : B1, O, lm, st);
}

template <bool LOWRANK, int G>
int launch_t(GramRows P, cudaStream_t s) {
    const int n = P.fa.n, pitch = LOWRANK ? RowAddr::pitch(n) : gram_pitch(P.fa);
    // vectors per CTA: up to 16 while the two buffers stay within 64 KB (3 CTAs per SM),
    // at least the K planes of one batch item
    const int most = std::max(1, std::min<int>(16, 64 * 1024 / (2 * pitch * (int)sizeof(float2))));
    const int per = !LOWRANK ? 1 : P.K;
    P.nbv = std::max(1, std::min(P.batch, most / per));
    P.V = P.nbv * per;
    P.nbg = (P.batch + P.nbv - 1) / P.nbv;
    const size_t smem = (size_t)2 * P.V * pitch * sizeof(float2);
    const int64_t blocks = (int64_t)P.nbg * (!LOWRANK ? P.K : 1) * P.rows * P.nseg;
    P.T = streams(P.fa, P.V, smem, blocks, 16);
    P.dt = Div(P.T);
    P.dbg = Div(P.nbg);
    P.dk = Div(P.K);
    P.drow = Div(P.rows);
    if (P.V * P.T > kMaxThreads) return fail(PFB_ERR_UNSUPPORTED, "Gram rows: too many threads");
    if (blocks >= (1LL << 31)) return fail(PFB_ERR_UNSUPPORTED, "too many vectors for the fused FFT");
    auto k = gram_rows_kernel<LOWRANK, G>;
    PFB_RAISE_SMEM(k, (int)smem);
    k<<<(unsigned)blocks, P.V * P.T, smem, s>>>(P);
    PFB_CHECK_LAUNCH();
    return PFB_OK;
}

template <int G>
int launch_gram_rows_t(const GramRows &P, cudaStream_t s) {
    return P.lowrank ? launch_t<true, G>(P, s) : launch_t<false, G>(P, s);
}

}  // namespace fft
}  // namespace pfb
