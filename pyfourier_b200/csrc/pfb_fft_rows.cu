// Row passes of the fused FFT: transforms along x, lanes along the butterflies of a
// vector so that the accesses along x are coalesced (see pfb_fft.cuh).
#include "pfb_fft_passes.cuh"

namespace pfb {
namespace fft {
namespace {

// forward: rows of T (N0 long, [plane][kz][ky][x]) -> the interleaved grid
// [grp][kz][ky][kx][ch].  A CTA holds cpt channels of kpt rows ky of one (grp, kz), so
// that what it writes is whole runs of channels (all of a row's memory when it holds all channels);
// the transform leaves through shared memory, channels side by side.
template <int G>
__global__ void __launch_bounds__(kMaxThreads, min_blocks(big_group(G))) row_fwd_kernel(const RowPass P) {
    extern __shared__ __align__(16) float2 fsm[];
    using A = RowAddr;
    const int n = P.fa.n, T = P.T, N0 = P.N0;
    int stream;
    const int v = P.dt.split(threadIdx.x, stream);
    const A ad{v * A::pitch(n)};
    float2 *b0 = fsm, *b1 = fsm + P.buf;
    int cc, yb, kz, c;
    const int grp = P.dz.split(P.dyb.split(P.dchunk.split(blockIdx.x, cc), yb), kz);
    const int c0 = cc * P.cpt, ky0 = yb * P.kpt;
    const int nc = min(P.cpt, P.nch - c0), ny = min(P.kpt, P.nos1 - ky0);
    const int yl = P.dcpt.split(v, c);
    const bool on = c < nc && yl < ny;
    const float2 *src =
        on ? P.src + ((((int64_t)grp * P.nch + c0 + c) * P.nos2 + kz) * P.nos1 + ky0 + yl) * N0 : nullptr;
    const int hn = N0 / 2;
    auto ld = [&](int p) {
        const int x = (int)min((unsigned)(p + hn), (unsigned)(p + hn - n));  // mod n
        return on && x < N0 ? __ldg(src + x) : make_float2(0.f, 0.f);
    };
    // the buffer that the last stage does not read takes the result, [yl][kx][c]
    float2 *out = P.fa.nst % 2 == 0 ? b1 : b0;
    const int cp = P.cp;
    auto st = [&](int k, float2 r) {
        if (on) out[(yl * n + k) * cp + c] = r;
    };
    run<G>(P.fa, stream, T, ad, b0, b1, ld, st);
    __syncthreads();
    // copy-out: a thread keeps its unit (a channel, or a pair where that is 16-byte aligned)
    // and walks kx
    const bool pair = P.nch % 2 == 0 && nc % 2 == 0 && c0 % 2 == 0;
    const int nu = pair ? nc / 2 : nc;
    const bool full = nu == P.dunit.d;
    const int kx0 = full ? P.dunit(threadIdx.x) : threadIdx.x / nu, un = threadIdx.x - kx0 * nu;
    const int step = full ? P.dunit(blockDim.x) : blockDim.x / nu;
    if (kx0 >= step) return;
    for (int y = 0; y < ny; ++y) {
        float2 *d = P.dst + ((int64_t)grp * P.gvol + ((int64_t)kz * P.nos1 + ky0 + y) * n) * P.nch + c0;
        const float2 *o = out + y * n * cp;
        if (pair) {
            for (int kx = kx0; kx < n; kx += step) {
                const float2 a = o[kx * cp + 2 * un], b = o[kx * cp + 2 * un + 1];
                *reinterpret_cast<float4 *>(d + (int64_t)kx * P.nch + 2 * un) = make_float4(a.x, a.y, b.x, b.y);
            }
        } else {
            for (int kx = kx0; kx < n; kx += step) d[(int64_t)kx * P.nch + un] = o[kx * cp + un];
        }
    }
}

// inverse: rows of the planar grid (n long) -> rows of T cropped to N0
template <int G>
__global__ void __launch_bounds__(kMaxThreads, min_blocks(big_group(G))) row_inv_kernel(const RowPass P) {
    extern __shared__ __align__(16) float2 fsm[];
    using A = RowAddr;
    const int n = P.fa.n, T = P.T;
    int stream;
    const int v = P.dt.split(threadIdx.x, stream);
    const A ad{v * A::pitch(n)};
    const int64_t u = (int64_t)blockIdx.x * P.V + v;
    const bool on = u < P.nvec;
    const float2 *src = P.src + (on ? u : 0) * n;
    auto ld = [&](int p) { return __ldg(src + p); };
    float2 *dst = P.dst + u * P.N0;
    const int hn = P.N0 / 2;
    auto st = [&](int k, float2 r) {
        const int c = k ? n - k + hn : hn;
        const int o = (int)min((unsigned)c, (unsigned)(c - n));  // mod n
        if (on && o < P.N0) dst[o] = r;
    };
    run<G>(P.fa, stream, T, ad, fsm, fsm + P.buf, ld, st);
}

// Vectors per CTA: 16, or 8 where two buffers of 16 take more than 48 KB (fewer than 4
// CTAs per SM) or the pass has too few vectors to fill the chip
int vectors(int n, int64_t nvec) {
    return 2 * 16 * RowAddr::pitch(n) * (int)sizeof(float2) > 48 * 1024 || nvec < 16 * 296 ? 8 : 16;
}

template <int G>
int launch_fwd(RowPass P, cudaStream_t s) {
    const int n = P.fa.n, most = vectors(n, P.nvec);
    // channels per tile: all of them up to `most`, else the most even split (in pairs when
    // there are pairs); rows ky fill up, and the CTA has just the vectors it uses
    const int chunks = (P.nch + most - 1) / most;
    P.cpt = (P.nch + chunks - 1) / chunks;
    if (P.nch % 2 == 0 && chunks > 1) P.cpt += P.cpt & 1;
    P.nchunk = (P.nch + P.cpt - 1) / P.cpt;
    P.kpt = P.nchunk > 1 ? 1 : std::min(most / P.cpt, P.nos1);
    P.nyb = (P.nos1 + P.kpt - 1) / P.kpt;
    P.V = P.cpt * P.kpt;
    P.cp = P.cpt >= 8 ? P.cpt | 1 : P.cpt;  // odd pitch from 8 channels: conflict-free transposes
    P.buf = std::max(P.V * RowAddr::pitch(n), P.kpt * n * P.cp);
    const size_t smem = (size_t)2 * P.buf * sizeof(float2);
    const int64_t ngrp = P.nvec / ((int64_t)P.nch * P.nos1 * P.nos2);
    const int64_t blocks = ngrp * P.nos2 * P.nyb * P.nchunk;
    P.T = streams(P.fa, P.V, smem, blocks, 16);
    P.dt = Div(P.T);
    P.dchunk = Div(P.nchunk);
    P.dyb = Div(P.nyb);
    P.dz = Div(P.nos2);
    P.dcpt = Div(P.cpt);
    P.dunit = Div(P.nch % 2 == 0 && P.cpt % 2 == 0 ? P.cpt / 2 : P.cpt);
    if (blocks >= (1LL << 31)) return fail(PFB_ERR_UNSUPPORTED, "too many vectors for the fused FFT");
    auto k = row_fwd_kernel<G>;
    PFB_RAISE_SMEM(k, (int)smem);
    k<<<(unsigned)blocks, P.V * P.T, smem, s>>>(P);
    PFB_CHECK_LAUNCH();
    return PFB_OK;
}

template <int G>
int launch_inv(RowPass P, cudaStream_t s) {
    P.V = P.fa.n > 128 ? 8 : vectors(P.fa.n, P.nvec);
    P.buf = P.V * RowAddr::pitch(P.fa.n);
    const size_t smem = (size_t)(P.fa.nst > 2 ? 2 : 1) * P.buf * sizeof(float2);
    const int64_t blocks = (P.nvec + P.V - 1) / P.V;
    P.T = streams(P.fa, P.V, smem, blocks, 16);
    P.dt = Div(P.T);
    if (blocks >= (1LL << 31)) return fail(PFB_ERR_UNSUPPORTED, "too many vectors for the fused FFT");
    auto k = row_inv_kernel<G>;
    PFB_RAISE_SMEM(k, (int)smem);
    k<<<(unsigned)blocks, P.V * P.T, smem, s>>>(P);
    PFB_CHECK_LAUNCH();
    return PFB_OK;
}

}  // namespace

int launch_row(const RowPass &P, bool inv, cudaStream_t s) {
    if (P.nvec == 0) return PFB_OK;
    const int st = launch_row_tma(P, inv, s);
    if (st) return st == 1 ? PFB_OK : st;
    switch (plan_group(P.fa)) {
        case 0: return inv ? launch_inv<0>(P, s) : launch_fwd<0>(P, s);
        case 1: return inv ? launch_inv<1>(P, s) : launch_fwd<1>(P, s);
        case 2: return inv ? launch_inv<2>(P, s) : launch_fwd<2>(P, s);
        default: return inv ? launch_inv<3>(P, s) : launch_fwd<3>(P, s);
    }
}

}  // namespace fft
}  // namespace pfb
