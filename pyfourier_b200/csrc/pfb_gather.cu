// Interpolation from the channel-interleaved grid, and the trajectory gradient: the
// gather half of the pipeline (src/pyfourier/_subroutines/_grid/_cart2noncart, and the
// analytic derivative for _nufft/_nufft.py:175-209).
//
// In the interleaved grid the taps of one x row of a sample's kernel box are W x
// channels consecutive values, so the unit of work is the x row: U lanes hold one row
// (lane = x tap x channel, 16-byte channel pairs when the channel count is even), a warp
// holds S = 32 / U consecutive bin-sorted samples side by side, and every lane walks the
// W^(D-1) rows of its sample with its y and z weights and offsets in registers: per row
// one address add, one load and one packed FMA per channel.  The x weights are applied
// once, after the rows, and the W lanes of a channel are added by shuffles.  Channels
// past one warp-wide row are taken in further chunks of the same sample.
//
// This replaced one warp per sample with lanes = channels x tap groups over a tap list in
// shared memory (and, at 32 channels of width 4, x rows in shared memory): with few
// channels that spent its time building the list and left 3 of 4 lanes' loads
// uncoalesced, and widths 5 to 7 walked 8^D taps.
//
// Measured (interp of 1.2 M radial samples, 3D width 4, us, before / now): 1 channel 427 /
// 98, 4 channels 453 / 172, 8 channels 559 / 302, 16 channels 801 / 563; 2D width 4, 205 k
// samples: 1 channel 90 / 13, 8 channels 109 / 43; 3D width 6, 384 k samples, 8 channels
// 951 / 349.
#include "pfb_common.cuh"

namespace pfb {
namespace {

constexpr int kWarps = 8;      // warps per CTA
constexpr int kMaxSlots = 8;   // samples side by side in a warp

struct Gather {
    Geom g;
    const float *cos0, *cos1, *cos2;  // sorted grid coordinates (gradient weights)
    const int *sframe, *perm;
    const float *rec;          // plan records of tap_rec(D, WM) words
    int64_t mtot;
    const float2 *grid;        // interleaved
    float2 *res;               // [M][nch]
    Chan ch;
    int nu;                    // units (V channels) per grid point
    int cpv, nchunk;           // units per x tap of a chunk, chunks
    int U, S;                  // lanes per sample, samples per warp
    // trajectory gradient
    const float2 *vt;          // [M][B] values (weight applied)
    const float2 *basis, *tB;
    const int64_t *frame_off;
    int readout;
    float chain[kMaxDim];
    float *grad;               // (M, ndim) in original sample order
    int accumulate;
};

template <int V>
struct Unit;
template <>
struct Unit<1> {
    using T = float2;
    static __device__ __forceinline__ void fma(float w, T v, float2 (&a)[1]) {
        a[0] = __ffma2_rn(make_float2(w, w), v, a[0]);
    }
};
template <>
struct Unit<2> {
    using T = float4;
    static __device__ __forceinline__ void fma(float w, T v, float2 (&a)[2]) {
        const float2 ww = make_float2(w, w);
        a[0] = __ffma2_rn(ww, make_float2(v.x, v.y), a[0]);
        a[1] = __ffma2_rn(ww, make_float2(v.z, v.w), a[1]);
    }
};

// FFT-layout position of first tap x0 in [0, nos), and of the tap i places after
// position q (i < w <= nos, so one wrap is enough; the smaller of the two as unsigned
// numbers is the one inside the grid)
__device__ __forceinline__ int first_pos(int x0, int sh, int nos) {
    const int q = x0 - sh;
    return q < 0 ? q + nos : q;
}
__device__ __forceinline__ int tap_pos(int q, int i, int nos) {
    return (int)min((unsigned)(q + i), (unsigned)(q + i - nos));
}

// gradient weight (kernel value) and derivative of tap t on axis a of sorted sample j
__device__ __forceinline__ void grad_weight(const Gather &P, int j, int jend, int a, int t, float *w,
                                            float *d) {
    float wv = 0.f, dv = 0.f;
    if (j < jend && t < P.g.w[a]) {
        if (P.g.cart[a]) {
            wv = 1.f;
        } else {
            const float c = (a == 0 ? P.cos0 : (a == 1 ? P.cos1 : P.cos2))[j];
            const float halfw = 0.5f * (float)P.g.w[a];
            float k;
            wv = kb_eval_deriv(((float)(start_index(c, P.g.w[a], 0) + t) - c) / halfw, P.g.beta[a], &k);
            dv = -k / halfw;
        }
    }
    *w = wv;
    *d = dv;
}

// adds Re(conj(d_a) v) of channel c of sample j: d_a times the channel factor B_l(t)
// basis[f, k], v the channel's value
template <int D>
__device__ __forceinline__ void grad_add(const Gather &P, int j, int f, int c, float2 d0, float2 d1, float2 d2,
                                         float (&g)[3]) {
    int b = c;
    float2 fac = make_float2(1.f, 0.f);
    if (P.ch.K || P.tB) {
        const int Kc = P.ch.K ? P.ch.K : 1;
        const int kk = c % Kc, lb = c / Kc, l = lb / P.ch.B;
        b = lb - l * P.ch.B;
        if (P.tB) fac = P.tB[(int64_t)l * P.readout + (int)((P.perm[j] - P.frame_off[f]) % P.readout)];
        if (P.ch.K) fac = cmul(fac, P.basis[(int64_t)f * P.ch.K + kk]);
    }
    const float2 v = __ldg(P.vt + (int64_t)j * P.ch.B + b);
    d0 = cmul(d0, fac);
    g[0] += d0.x * v.x + d0.y * v.y;
    if (D > 1) {
        d1 = cmul(d1, fac);
        g[1] += d1.x * v.x + d1.y * v.y;
    }
    if (D > 2) {
        d2 = cmul(d2, fac);
        g[2] += d2.x * v.x + d2.y * v.y;
    }
}

// WM: taps per axis of the plan records; V channels per lane; WIDE: 64-bit element
// offsets; GRAD: the trajectory gradient instead of the interpolation; NC chunks of
// channels per pass over the rows.
// Registers: 8 to 16 row loads in flight per lane at 3 CTAs (24 warps) per SM.
template <int D, int WM, int V, bool WIDE, bool GRAD, int NC>
__global__ void __launch_bounds__(kWarps * 32, GRAD && D == 3 ? 2 : 3) gather_rows_kernel(const Gather P) {
    using T = typename Unit<V>::T;
    using Off = typename std::conditional<WIDE, int64_t, int>::type;
    constexpr int REC = tap_rec(D, WM), DW = D * WM;
    constexpr int NPRE = (kMaxSlots * REC + 31) / 32 < 4 ? (kMaxSlots * REC + 31) / 32 : 4;
    constexpr int WY = D > 1 ? WM : 1, WZ = D > 2 ? WM : 1;
    constexpr int ZU = WM == 4 ? (V * NC == 1 ? 4 : (V * NC == 2 ? 2 : 1)) : 1;  // z rows unrolled
    __shared__ __align__(16) float s_rec[kWarps][NPRE * 32];
    __shared__ float s_w[GRAD ? kWarps : 1][GRAD ? kMaxSlots * DW : 1];
    __shared__ float s_d[GRAD ? kWarps : 1][GRAD ? kMaxSlots * DW : 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cpv = P.cpv, U = P.U, S = P.S, nch = P.ch.nch;
    const int slot = lane / U, e = lane - slot * U;
    const int ix = e / cpv, cu = e - ix * cpv;
    const bool active = slot < S;
    const int w0 = P.g.w[0], w1 = D > 1 ? P.g.w[1] : 1, w2 = D > 2 ? P.g.w[2] : 1;
    // each CTA takes a contiguous run of bin-sorted samples: its warps gather from the
    // same few tiles, which stay in L1
    const int mtot = (int)P.mtot;  // a plan has less than 2^31 samples
    const int per = (int)((P.mtot + gridDim.x - 1) / gridDim.x);
    const int jbeg = (int)min((int64_t)blockIdx.x * per, P.mtot), jend = jbeg + min(per, mtot - jbeg);
    // the records and frame of the warp's next samples are loaded into registers while
    // the current ones gather
    float pre[NPRE];
    int pf = 0;
    // a warp takes NB consecutive samples, S at a time; the gradient evaluates the weights
    // and derivatives of all of them at once, so that every lane has some
    const int NB = GRAD ? kMaxSlots : S;
    auto fetch = [&](int j0, int jlim) {
        const int left = min(jlim - j0, S);  // <= 0 past the CTA's samples
        const float *rec = P.rec + (int64_t)j0 * REC + lane;
#pragma unroll
        for (int k = 0; k < NPRE; ++k) pre[k] = lane + 32 * k < left * REC ? __ldg(rec + 32 * k) : 0.f;
        pf = (!P.ch.K || GRAD) && slot < left ? P.sframe[j0 + slot] : 0;
    };
    fetch(jbeg + warp * NB, min(jend, jbeg + warp * NB + NB));
    for (int jb = jbeg + warp * NB, j0 = jb; jb < jend;) {
        const int jlim = min(jend, jb + NB);
#pragma unroll
        for (int k = 0; k < NPRE; ++k) s_rec[warp][lane + 32 * k] = pre[k];
        const int frame = pf, grp = P.ch.K ? 0 : pf;
        const int sb = GRAD ? j0 - jb : 0;  // first sample's place among the warp's NB
        if (GRAD && sb == 0) {
            // weights and their derivatives: one (sample, axis, tap) per lane and turn
            for (int i = lane; i < NB * DW; i += 32) {
                const int sl = i / DW, r = i - sl * DW, a = r / WM, t = r - a * WM;
                grad_weight(P, jb + sl, jend, a, t, &s_w[warp][i], &s_d[warp][i]);
            }
        }
        __syncwarp();
        const int j = j0 + slot;
        const bool valid = active && j < jlim;
        j0 += S;
        if (j0 >= jlim) {
            jb += kWarps * NB;
            j0 = jb;
        }
        fetch(j0, min(jend, jb + NB));
        const float *r = s_rec[warp] + (valid ? slot * REC : 0);
        const int *x0 = reinterpret_cast<const int *>(r) + DW;
        const float *rw = GRAD ? s_w[warp] + (valid ? (sb + slot) * DW : 0) : r;
        const float *rd = GRAD ? s_d[warp] + (valid ? (sb + slot) * DW : 0) : r;
        const float wx = rw[ix < WM ? ix : 0];
        const Off xo = (Off)tap_pos(first_pos(x0[0], P.g.sh[0], P.g.nos[0]), valid ? ix : 0, P.g.nos[0]) * P.nu;
        float wy[WY], dy[GRAD ? WY : 1];
        Off yo[WY];
        const int qy = D > 1 ? first_pos(x0[D > 1 ? 1 : 0], P.g.sh[1], P.g.nos[1]) : 0;
        const int qz = D > 2 ? first_pos(x0[D > 2 ? 2 : 0], P.g.sh[2], P.g.nos[2]) : 0;
        const Off sy1 = (Off)P.g.nos[0] * P.nu, sz1 = sy1 * P.g.nos[1];
#pragma unroll
        for (int i = 0; i < WY; ++i) {
            wy[i] = D > 1 ? rw[WM + i] : 1.f;
            if constexpr (GRAD) dy[i] = D > 1 ? rd[WM + i] : 0.f;
            yo[i] = D > 1 ? (Off)tap_pos(qy, i < w1 ? i : 0, P.g.nos[1]) * sy1 : 0;
        }
        const T *G = reinterpret_cast<const T *>(P.grid + (int64_t)grp * P.g.gvol * nch);
        float gacc[3] = {0.f, 0.f, 0.f};
        // the gradient's place and old value, read ahead of the gathers
        int64_t go = 0;
        float g0[GRAD ? D : 1] = {0.f};
        if (GRAD && valid && e == 0) {
            go = (int64_t)P.perm[j] * D;
#pragma unroll
            for (int a = 0; a < (GRAD ? D : 1); ++a) g0[a] = P.accumulate ? P.grad[go + a] : 0.f;
        }
        for (int q0 = 0; q0 < P.nchunk; q0 += NC) {
            // taps past an axis's width have weight 0 and repeat tap 0's address: no branch
            // between the loads of a pass, so all of them are in flight together
            float2 s0[NC][V], sy[NC][V], sz[NC][V];
#pragma unroll
            for (int n = 0; n < NC; ++n)
#pragma unroll
                for (int k = 0; k < V; ++k) s0[n][k] = sy[n][k] = sz[n][k] = make_float2(0.f, 0.f);
            if (valid) {
                const T *Gq[NC];
#pragma unroll
                for (int n = 0; n < NC; ++n) {
                    // past the last chunk or channel: the sample's first unit (result discarded)
                    const int cq = (q0 + n) * cpv + cu;
                    Gq[n] = G + xo + (cq < P.nu ? cq : 0);
                }
#pragma unroll ZU
                for (int iz = 0; iz < WZ; ++iz) {
                    Off zo = 0;
                    if (D > 2) zo = (Off)tap_pos(qz, iz < w2 ? iz : 0, P.g.nos[2]) * sz1;
                    T v[NC][WY];
#pragma unroll
                    for (int iy = 0; iy < WY; ++iy)
#pragma unroll
                        for (int n = 0; n < NC; ++n) v[n][iy] = __ldg(Gq[n] + (zo + yo[iy]));
                    const float wz = D > 2 ? rw[2 * WM + iz] : 1.f;
                    const float2 wz2 = make_float2(wz, wz);
#pragma unroll
                    for (int n = 0; n < NC; ++n) {
                        float2 a[V], b[V];
#pragma unroll
                        for (int k = 0; k < V; ++k) a[k] = b[k] = make_float2(0.f, 0.f);
#pragma unroll
                        for (int iy = 0; iy < WY; ++iy) {
                            Unit<V>::fma(wy[iy], v[n][iy], a);
                            if constexpr (GRAD && D > 1) Unit<V>::fma(dy[iy], v[n][iy], b);
                        }
#pragma unroll
                        for (int k = 0; k < V; ++k) {
                            s0[n][k] = __ffma2_rn(wz2, a[k], s0[n][k]);
                            if constexpr (GRAD) {
                                if (D > 1) sy[n][k] = __ffma2_rn(wz2, b[k], sy[n][k]);
                                if (D > 2) {
                                    const float dz = rd[2 * WM + iz];
                                    sz[n][k] = __ffma2_rn(make_float2(dz, dz), a[k], sz[n][k]);
                                }
                            }
                        }
                    }
                }
            }
#pragma unroll
            for (int n = 0; n < NC; ++n) {
            const int cq = (q0 + n) * cpv + cu;
            const bool on = valid && cq < P.nu;
            if constexpr (!GRAD) {
                const float2 wx2 = make_float2(wx, wx);
#pragma unroll
                for (int k = 0; k < V; ++k) s0[n][k] = __fmul2_rn(wx2, s0[n][k]);
                // add the w0 lanes (cpv apart) of each channel into the lane of tap 0
                for (int m = w0; m > 1;) {
                    const int h = (m + 1) >> 1;
                    const bool add = ix < m - h;
#pragma unroll
                    for (int k = 0; k < V; ++k) {
                        const float tx = __shfl_down_sync(0xffffffffu, s0[n][k].x, h * cpv);
                        const float ty = __shfl_down_sync(0xffffffffu, s0[n][k].y, h * cpv);
                        if (add) s0[n][k] = make_float2(s0[n][k].x + tx, s0[n][k].y + ty);
                    }
                    m = h;
                }
                if (on && ix == 0) {
                    T *dst = reinterpret_cast<T *>(P.res + (int64_t)j * nch) + cq;
                    if constexpr (V == 1) *dst = s0[n][0];
                    else *dst = make_float4(s0[n][0].x, s0[n][0].y, s0[n][V - 1].x, s0[n][V - 1].y);
                }
            } else if (on) {
                const float dx = rd[ix < WM ? ix : 0];
#pragma unroll
                for (int k = 0; k < V; ++k) {
                    const float2 wx2 = make_float2(wx, wx);
                    grad_add<D>(P, j, frame, cq * V + k, __fmul2_rn(make_float2(dx, dx), s0[n][k]),
                                __fmul2_rn(wx2, sy[n][k]), __fmul2_rn(wx2, sz[n][k]), gacc);
                }
            }
            }
        }
        if constexpr (GRAD) {
            // add the sample's U lanes
            for (int n = U; n > 1;) {
                const int h = (n + 1) >> 1;
                const bool add = e < n - h;
#pragma unroll
                for (int a = 0; a < D; ++a) {
                    const float t = __shfl_down_sync(0xffffffffu, gacc[a], h);
                    if (add) gacc[a] += t;
                }
                n = h;
            }
            if (valid && e == 0) {
#pragma unroll
                for (int a = 0; a < D; ++a) P.grad[go + a] = g0[a] + gacc[a] * P.chain[a];
            }
        }
        __syncwarp();
    }
}

// The gather with a channel per lane (many channels, see launch_t): one warp per sample.
// Lanes write one record per x row (the row's y / z offset and its weight w_y * w_z; with
// GRAD also the two products with one derivative) and the x positions into shared memory;
// the rows' gathers go out RB rows at a time, each x column accumulates over the rows and
// the columns are combined with the x weights once per sample.  CH: the channel count when
// fixed at compile time: a row whose x taps are not split by the fftshift seam is then one
// pointer and its taps sit at fixed offsets from it (3D 200^3, 32 channels, width 4: at 94 %
// of the L1 data pipe; the form above, which takes 32 channels in two chunks of 16, ran
// 6.64 ms against 5.13 ms).
template <int D, int WM, bool WIDE, int CH, bool GRAD>
__global__ void __launch_bounds__(kWarps * 32, GRAD ? 2 : 3) gather_xrow_kernel(const Gather P) {
    constexpr int NR = D == 3 ? WM * WM : (D == 2 ? WM : 1), REC = tap_rec(D, WM), DW = D * WM;
    constexpr int RB = D == 1 ? 1 : (WM == 4 ? 4 : 2);  // rows in flight
    constexpr int NG = GRAD && D > 1 ? NR : 1;
    constexpr bool GY = GRAD && D > 1, GZ = GRAD && D > 2;  // gradients besides x
    constexpr int NW = (NR + 31) / 32;
    constexpr int NB = GRAD ? 32 / DW : 1;  // consecutive samples of a warp (gradient weights of all at once)
    static_assert(REC <= 32 && NR % RB == 0, "one record word per lane, whole batches of rows");
    __shared__ __align__(16) float s_rec[kWarps][32];
    __shared__ __align__(16) int s_px[kWarps][8];
    __shared__ __align__(16) int s_roff[kWarps][NR];
    __shared__ __align__(16) float2 s_rw[kWarps][NR];
    __shared__ __align__(16) float2 s_ry[kWarps][NG], s_rz[kWarps][D > 2 ? NG : 1];  // (dy wz), (wy dz)
    __shared__ float s_w[kWarps][GRAD ? NB * DW : 1], s_d[kWarps][GRAD ? NB * DW : 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nch = CH ? CH : P.ch.nch;
    const int mtot = (int)P.mtot;  // a plan has less than 2^31 samples
    const int per = (int)((P.mtot + gridDim.x - 1) / gridDim.x);
    const int jbeg = (int)min((int64_t)blockIdx.x * per, P.mtot), jend = jbeg + min(per, mtot - jbeg);
    float pre = 0.f;
    int pf = 0, pg = 0;
    auto fetch = [&](int j) {
        if (j < jend) {
            if (lane < REC) pre = __ldg(P.rec + (int64_t)j * REC + lane);
            pf = P.ch.K && !GRAD ? 0 : P.sframe[j];
            if (GRAD) pg = P.perm[j];
        }
    };
    fetch(jbeg + warp * NB);
    for (int jb = jbeg + warp * NB, j = jb; j < jend;) {
        const int sb = GRAD ? j - jb : 0;
        s_rec[warp][lane] = pre;
        if constexpr (GRAD)
            if (sb == 0 && lane < NB * DW) {
                const int sl = lane / DW, q = lane - sl * DW;
                grad_weight(P, jb + sl, jend, q / WM, q % WM, &s_w[warp][lane], &s_d[warp][lane]);
            }
        const int frame = pf, grp = P.ch.K ? 0 : pf;
        // the gradient's place and old value, read ahead of the gathers
        const int64_t go = (int64_t)pg * D + lane;
        const float g0 = GRAD && P.accumulate && lane < D ? P.grad[go] : 0.f;
        const int jn = !GRAD ? j + kWarps : (sb + 1 < NB && j + 1 < jend ? j + 1 : jb + kWarps * NB);
        fetch(jn);
        __syncwarp();
        const float *r = s_rec[warp];
        const int *x0 = reinterpret_cast<const int *>(r) + DW;
        const float *rw = GRAD ? s_w[warp] + sb * DW : r, *rd = GRAD ? s_d[warp] + sb * DW : r;
        if (lane < WM)  // taps past the width repeat tap 0's position (weight 0)
            s_px[warp][lane] =
                tap_pos(first_pos(x0[0], P.g.sh[0], P.g.nos[0]), lane < P.g.w[0] ? lane : 0, P.g.nos[0]);
#pragma unroll
        for (int k = 0; k < NW; ++k) {
            const int t = lane + 32 * k;
            if (t < NR) {
                const int iy = t % WM, iz = t / WM;
                const bool ok = D == 1 || (iy < P.g.w[1] && (D < 3 || iz < P.g.w[2]));
                float w = D == 1 ? 1.f : 0.f, wy = 0.f, wz = 0.f;
                int off = 0;
                if (D > 1 && ok) {
                    const float vz = D > 2 ? rw[2 * WM + iz] : 1.f;
                    w = rw[WM + iy] * vz;
                    if (GY) wy = rd[WM + iy] * vz;
                    if (GZ) wz = rw[WM + iy] * rd[2 * WM + iz];
                    off = tap_pos(first_pos(x0[D > 1 ? 1 : 0], P.g.sh[1], P.g.nos[1]), iy, P.g.nos[1]) * P.g.nos[0];
                    if (D > 2)
                        off += tap_pos(first_pos(x0[D > 2 ? 2 : 0], P.g.sh[2], P.g.nos[2]), iz, P.g.nos[2]) *
                               (P.g.nos[0] * P.g.nos[1]);
                    if (!WIDE) off *= nch;
                }
                s_roff[warp][t] = off;
                s_rw[warp][t] = make_float2(w, w);
                if constexpr (GY) s_ry[warp][t] = make_float2(wy, wy);
                if constexpr (GZ) s_rz[warp][t] = make_float2(wz, wz);
            }
        }
        __syncwarp();
        const float2 *G = P.grid + (int64_t)grp * P.g.gvol * nch;
        float gacc[3] = {0.f, 0.f, 0.f};
        for (int c0 = 0; c0 < nch; c0 += 32) {
            const int c = c0 + lane;
            const float2 *Gc = G + (c < nch ? c : nch - 1);  // in-bounds address; result discarded
            int px[WM];
            if constexpr (WM == 4) {
                const int4 p4 = *reinterpret_cast<const int4 *>(s_px[warp]);
                px[0] = p4.x, px[1] = p4.y, px[2] = p4.z, px[3] = p4.w;
            } else {
#pragma unroll
                for (int u = 0; u < WM; ++u) px[u] = s_px[warp][u];
            }
            float2 ax[WM], bx[GY ? WM : 1], cx[GZ ? WM : 1];
#pragma unroll
            for (int u = 0; u < WM; ++u) {
                ax[u] = make_float2(0.f, 0.f);
                if constexpr (GY) bx[u] = ax[u];
                if constexpr (GZ) cx[u] = ax[u];
            }
            auto run = [&](auto addr) {
#pragma unroll
                for (int rb = 0; rb < NR / RB; ++rb) {
                    float2 v[RB * WM];
                    int o[RB];
                    if constexpr (RB == 4) {
                        const int4 o4 = reinterpret_cast<const int4 *>(s_roff[warp])[rb];
                        o[0] = o4.x, o[1] = o4.y, o[2] = o4.z, o[3] = o4.w;
                    } else if constexpr (RB == 2) {
                        const int2 o2 = reinterpret_cast<const int2 *>(s_roff[warp])[rb];
                        o[0] = o2.x, o[1] = o2.y;
                    } else {
                        o[0] = 0;  // 1D: the one row
                    }
#pragma unroll
                    for (int q = 0; q < RB; ++q) {
#pragma unroll
                        for (int u = 0; u < WM; ++u) v[q * WM + u] = __ldg(addr(o[q], u));
                    }
#pragma unroll
                    for (int q = 0; q < RB; ++q) {
                        const float2 wr = s_rw[warp][rb * RB + q];
#pragma unroll
                        for (int u = 0; u < WM; ++u) ax[u] = __ffma2_rn(wr, v[q * WM + u], ax[u]);
                        if constexpr (GY) {
                            const float2 wy = s_ry[warp][rb * RB + q];
#pragma unroll
                            for (int u = 0; u < WM; ++u) bx[u] = __ffma2_rn(wy, v[q * WM + u], bx[u]);
                        }
                        if constexpr (GZ) {
                            const float2 wz = s_rz[warp][rb * RB + q];
#pragma unroll
                            for (int u = 0; u < WM; ++u) cx[u] = __ffma2_rn(wz, v[q * WM + u], cx[u]);
                        }
                    }
                }
            };
            // x taps side by side, not split by the seam (positions only step back there)
            if (CH > 0 && px[WM - 1] == px[0] + WM - 1) {
                const float2 *Gx0 = Gc + px[0] * CH;
                run([&](int o, int u) { return Gx0 + o + u * CH; });
            } else {
                const float2 *Gx[WM];
#pragma unroll
                for (int u = 0; u < WM; ++u) Gx[u] = WIDE ? Gc + (int64_t)px[u] * nch : Gc + px[u] * nch;
                run([&](int o, int u) { return WIDE ? Gx[u] + (int64_t)o * nch : Gx[u] + o; });
            }
            float2 d0 = make_float2(0.f, 0.f), d1 = d0, d2 = d0;
#pragma unroll
            for (int u = 0; u < WM; ++u) {
                const float w = u < P.g.w[0] ? (GRAD ? rd : rw)[u] : 0.f;
                d0 = __ffma2_rn(make_float2(w, w), ax[u], d0);
                if constexpr (GY) {
                    const float wx = u < P.g.w[0] ? rw[u] : 0.f;
                    d1 = __ffma2_rn(make_float2(wx, wx), bx[u], d1);
                    if constexpr (GZ) d2 = __ffma2_rn(make_float2(wx, wx), cx[u], d2);
                }
            }
            if (c < nch) {
                if constexpr (!GRAD) P.res[(int64_t)j * nch + c] = d0;
                else grad_add<D>(P, j, frame, c, d0, d1, d2, gacc);
            }
        }
        if constexpr (GRAD) {
#pragma unroll
            for (int a = 0; a < D; ++a)
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) gacc[a] += __shfl_xor_sync(0xffffffffu, gacc[a], off);
            if (lane < D) {
                const float g = lane == 0 ? gacc[0] : (lane == 1 ? gacc[1] : gacc[2]);
                P.grad[go] = g0 + g * P.chain[lane];
            }
        }
        __syncwarp();
        if (!GRAD) {
            j += kWarps;
        } else {
            if (jn != j + 1) jb = jn;
            j = jn;
        }
    }
}

template <int D, int WM, bool GRAD>
int launch_xrow(const Gather &P, cudaStream_t s) {
    const bool wide = P.g.gvol * (int64_t)P.ch.nch >= (1LL << 31);
    const int64_t cta = kWarps * (GRAD ? 32 / (D * WM) : 1);  // samples of a CTA's turn
    const int64_t need = (P.mtot + cta - 1) / cta;
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(need, 148LL * 64));
    auto run = [&](auto k) { k<<<blocks, kWarps * 32, 0, s>>>(P); };
    if (wide) run(gather_xrow_kernel<D, WM, true, 0, GRAD>);
    else if (P.ch.nch == 32 && !GRAD) run(gather_xrow_kernel<D, WM, false, GRAD ? 0 : 32, GRAD>);
    else run(gather_xrow_kernel<D, WM, false, 0, GRAD>);
    PFB_CHECK_LAUNCH();
    return PFB_OK;
}

template <int D, int WM, bool GRAD>
int launch_t(Gather &P, cudaStream_t s) {
    // channel pairs per lane when the rows of the grid and of the results keep them
    // 16-byte aligned
    auto a16 = [](const void *q) { return ((uintptr_t)q & 15u) == 0; };
    const bool pair = P.ch.nch % 2 == 0 && a16(P.grid) && a16(P.res);
    const int w0 = P.g.w[0], V = pair ? 2 : 1;
    P.nu = P.ch.nch / V;
    // chunks of at most 32 / w0 units, as even as they go
    const int most = 32 / w0;
    P.nchunk = (P.nu + most - 1) / most;
    if constexpr (WM >= 4) {
        // a channel per lane above 16 channels, and where the rows take too many chunks, us as
        // rows / channel per lane.  1D, one row: more than one chunk (512 k samples, width 4, 24
        // channels 195 / 140; width 6, 16 channels 201 / 140, 31 channels 428 / 168).  2D: two
        // of widths 7 and 8 and of an odd count at widths 5 and 6 (512 k samples, width 8, 5
        // channels 264 / 407, 16 channels 401 / 426, 15 channels in four 612 / 425; width 6, 9
        // channels 258 / 276, 16 channels 320 / 287; width 4, 15 channels 207 / 196), and any
        // of the gradient (102 k samples, width 8, 16 channels 131 / 162).  3D: two (width 6, 15
        // channels 1114 / 857, 16 channels 733 / 857, width 4, 15 channels 775 / 890)
        const int most_chunks = D == 1 ? 1 : D == 3 ? 2 : GRAD ? 8 : WM == 8 || (WM == 6 && !pair) ? 2 : 1;
        if (P.ch.nch > 16 || P.nchunk > most_chunks) return launch_xrow<D, WM, GRAD>(P, s);
    }
    P.cpv = (P.nu + P.nchunk - 1) / P.nchunk;
    P.U = w0 * P.cpv;
    P.S = std::min(32 / P.U, kMaxSlots);
    // the records of a warp's samples are held in at most 4 registers a lane
    P.S = std::max(1, std::min(P.S, 4 * 32 / tap_rec(D, WM)));
    const int64_t cta = kWarps * (GRAD ? kMaxSlots : P.S);  // samples of a CTA's turn
    const int64_t need = (P.mtot + cta - 1) / cta;
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(need, 148LL * 64));
    const bool wide = P.g.gvol * (int64_t)P.nu >= (1LL << 31);
    // few rows in 2D: two chunks keep enough loads in flight (the gradient has no registers
    // left for the second one; 1D has one chunk)
    constexpr int NC1 = GRAD || (D == 1 && WM >= 4) ? 1 : 2, NC2 = D == 3 ? 1 : NC1;
    auto run = [&](auto k) { k<<<blocks, kWarps * 32, 0, s>>>(P); };
    if (pair && wide) run(gather_rows_kernel<D, WM, 2, true, GRAD, 1>);
    else if (wide) run(gather_rows_kernel<D, WM, 1, true, GRAD, 1>);
    else if (pair && P.nchunk > 1) run(gather_rows_kernel<D, WM, 2, false, GRAD, NC2>);
    else if (pair) run(gather_rows_kernel<D, WM, 2, false, GRAD, 1>);
    else if (P.nchunk > 1) run(gather_rows_kernel<D, WM, 1, false, GRAD, NC1>);
    else run(gather_rows_kernel<D, WM, 1, false, GRAD, 1>);
    PFB_CHECK_LAUNCH();
    return PFB_OK;
}

template <bool GRAD>
int launch(Gather &P, cudaStream_t s) {
    switch (P.g.ndim * 10 + wm_of(P.g)) {
        case 11: return launch_t<1, 1, GRAD>(P, s);
        case 14: return launch_t<1, 4, GRAD>(P, s);
        case 16: return launch_t<1, 6, GRAD>(P, s);
        case 18: return launch_t<1, 8, GRAD>(P, s);
        case 21: return launch_t<2, 1, GRAD>(P, s);
        case 24: return launch_t<2, 4, GRAD>(P, s);
        case 26: return launch_t<2, 6, GRAD>(P, s);
        case 28: return launch_t<2, 8, GRAD>(P, s);
        case 31: return launch_t<3, 1, GRAD>(P, s);
        case 34: return launch_t<3, 4, GRAD>(P, s);
        case 36: return launch_t<3, 6, GRAD>(P, s);
        default: return launch_t<3, 8, GRAD>(P, s);
    }
}

void fill(const pfb_plan *p, const Chan &c, const float2 *grid, Gather &P) {
    P.g = p->g;
    P.cos0 = p->d_cos[0];
    P.cos1 = p->d_cos[1];
    P.cos2 = p->d_cos[2];
    P.sframe = p->d_sframe;
    P.perm = p->d_perm;
    P.rec = p->d_wtap;
    P.mtot = p->mtot;
    P.grid = grid;
    P.ch = c;
}

}  // namespace

int launch_interp_il(const pfb_plan *p, const Chan &c, const float2 *grid, float2 *res, cudaStream_t s) {
    Gather P{};
    fill(p, c, grid, P);
    P.res = res;
    return launch<false>(P, s);
}

int launch_traj_il(const pfb_plan *p, const Chan &c, const float2 *grid, const float2 *vt, const float2 *basis,
                   const float2 *tB, float *grad, bool accumulate, cudaStream_t s) {
    Gather P{};
    fill(p, c, grid, P);
    P.vt = vt;
    P.basis = basis;
    P.tB = tB;
    P.frame_off = p->d_frame_off;
    P.readout = p->readout;
    for (int a = 0; a < kMaxDim; ++a) P.chain[a] = (float)p->g.nos[a] / (float)p->g.n[a];
    P.grad = grad;
    P.accumulate = accumulate ? 1 : 0;
    return launch<true>(P, s);
}

}  // namespace pfb
