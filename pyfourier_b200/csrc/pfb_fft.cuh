// Batched 1D transforms of the fused FFT passes: butterflies, stages and stage plans.
//
// A vector's transform is a mixed-radix Stockham autosort FFT (Govindaraju et al., "High
// performance discrete Fourier transforms on graphics processors", SC 2008): stage s with
// radix r and ns = product of the earlier radices reads x_q = src[i + q n / r], multiplies
// by exp(-2 pi i j q / (ns r)) (j = i mod ns), takes the r-point DFT and writes
// dst[(i - j) r + j + k ns].  The first stage reads its points straight from global memory
// and the last writes straight to it, so a two-stage transform touches shared memory twice
// per element and waits at one barrier (a staged tile, stage by stage in shared memory,
// touched it six times: the 250-point column passes ran at 3.9 - 5.1 TB/s that way).
//
// A CTA holds NV vectors; thread (v, stream) of vector v takes butterflies stream,
// stream + T, ... of every stage.  Lanes run along the vectors where neighbouring vectors
// are neighbours in memory (column passes) and along the butterflies where a vector's own
// elements are (row passes): both keep the global accesses of a warp in whole segments.
//
// Radices 2 to 16, and up to 32 as the first of two stages; a prime factor that this does
// not take runs as a stage of its own in shared memory, an O(r^2) DFT over the pairs
// x_q +- x_(r - q).  Inverse transforms run the forward one and
// read it reversed, IDFT(x)[k] = DFT(x)[(n - k) mod n].  Twiddles are computed in double
// precision on the host.
#pragma once

#include "pfb_common.cuh"

namespace pfb {
namespace fft {

// Largest primes of a prime stage: above kMaxPrime the O(r^2) stage loses to the library's
// transform, but for an outer axis of a 3D grid up to kMaxPrime3 (measured beside fused_takes).
constexpr int kMaxPrime = 127, kMaxPrime3 = 167;

// cos and sin of 2 pi m / n for m = 0..n-1, evaluated at compile time (Taylor series in
// double after reduction to the first eighth of the circle)
template <int N>
struct Roots {
    float c[N], s[N];
    static constexpr double series(double x, int first) {
        double t = first ? x : 1.0, r = t;
        for (int k = first + 2; k < 30; k += 2) {
            t *= -x * x / (double)(k * (k - 1));
            r += t;
        }
        return r;
    }
    constexpr Roots() : c(), s() {
        for (int m = 0; m < N; ++m) {
            // angle in eighths: 8 m / N = o + f, o the octant
            const int o = 8 * m / N;
            const double pi = 3.14159265358979323846;
            double co = 0, si = 0;
            switch (o) {
                case 0: { const double a = 2 * pi * m / N; co = series(a, 0); si = series(a, 1); break; }
                case 1: case 2: { const double a = 2 * pi * (4 * m - N) / (4.0 * N); co = -series(a, 1); si = series(a, 0); break; }
                case 3: case 4: { const double a = 2 * pi * (2 * m - N) / (2.0 * N); co = -series(a, 0); si = -series(a, 1); break; }
                case 5: case 6: { const double a = 2 * pi * (4 * m - 3 * N) / (4.0 * N); co = series(a, 1); si = -series(a, 0); break; }
                default: { const double a = 2 * pi * (m - N) / N; co = series(a, 0); si = series(a, 1); break; }
            }
            c[m] = (float)co;
            s[m] = (float)si;
        }
    }
};

// Complex add / subtract / scale-and-add as packed (re, im) FP32 instructions: the
// same roundings as the componentwise forms (a - b is b * -1 + a, the product exact).
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
// -i * a
__device__ __forceinline__ float2 cmi(float2 a) { return make_float2(a.y, -a.x); }
__device__ __forceinline__ float2 caxpy(float s, float2 a, float2 y) { return __ffma2_rn(make_float2(s, s), a, y); }

// forward r-point DFTs, b_k = sum_q a_q exp(-2 pi i q k / r), in place.  The general form
// is for primes: pairs t = x_q + x_(r - q), d = x_q - x_(r - q) give outputs k and r - k.
template <int R>
__device__ __forceinline__ void dft(float2 *a) {
    constexpr Roots<R> W;
    constexpr int H = (R - 1) / 2;
    float2 t[H], d[H];
#pragma unroll
    for (int q = 1; q <= H; ++q) {
        t[q - 1] = cadd(a[q], a[R - q]);
        d[q - 1] = csub(a[q], a[R - q]);
    }
    const float2 a0 = a[0];
#pragma unroll
    for (int q = 0; q < H; ++q) a[0] = cadd(a[0], t[q]);
#pragma unroll
    for (int k = 1; k <= H; ++k) {
        float2 p = a0, u = make_float2(0.f, 0.f);
#pragma unroll
        for (int q = 1; q <= H; ++q) {
            p = caxpy(W.c[q * k % R], t[q - 1], p);
            u = caxpy(W.s[q * k % R], d[q - 1], u);
        }
        a[k] = cadd(p, cmi(u));
        a[R - k] = csub(p, cmi(u));
    }
}

template <>
__device__ __forceinline__ void dft<1>(float2 *) {}

template <>
__device__ __forceinline__ void dft<2>(float2 *a) {
    const float2 t = a[1];
    a[1] = csub(a[0], t);
    a[0] = cadd(a[0], t);
}

template <>
__device__ __forceinline__ void dft<3>(float2 *a) {
    const float s = 0.86602540378443871f;  // sin(2 pi / 3)
    const float2 t = cadd(a[1], a[2]), d = csub(a[1], a[2]);
    const float2 m = caxpy(-0.5f, t, a[0]);
    const float2 u = make_float2(s * d.y, -s * d.x);  // -i s d
    a[0] = cadd(a[0], t);
    a[1] = cadd(m, u);
    a[2] = csub(m, u);
}

template <>
__device__ __forceinline__ void dft<4>(float2 *a) {
    const float2 t0 = cadd(a[0], a[2]), t1 = csub(a[0], a[2]);
    const float2 t2 = cadd(a[1], a[3]), t3 = cmi(csub(a[1], a[3]));
    a[0] = cadd(t0, t2);
    a[2] = csub(t0, t2);
    a[1] = cadd(t1, t3);
    a[3] = csub(t1, t3);
}

template <>
__device__ __forceinline__ void dft<5>(float2 *a) {
    // cos and sin of 2 pi / 5 and 4 pi / 5
    const float c1 = 0.30901699437494745f, c2 = -0.80901699437494734f;
    const float s1 = 0.95105651629515353f, s2 = 0.58778525229247325f;
    const float2 t1 = cadd(a[1], a[4]), t2 = cadd(a[2], a[3]);
    const float2 t3 = csub(a[1], a[4]), t4 = csub(a[2], a[3]);
    const float2 p1 = caxpy(c2, t2, caxpy(c1, t1, a[0]));
    const float2 p2 = caxpy(c1, t2, caxpy(c2, t1, a[0]));
    const float2 q1 = caxpy(s2, t4, make_float2(s1 * t3.x, s1 * t3.y));
    const float2 q2 = caxpy(-s1, t4, make_float2(s2 * t3.x, s2 * t3.y));
    a[0] = cadd(a[0], cadd(t1, t2));
    a[1] = cadd(p1, cmi(q1));
    a[4] = csub(p1, cmi(q1));
    a[2] = cadd(p2, cmi(q2));
    a[3] = csub(p2, cmi(q2));
}

template <>
__device__ __forceinline__ void dft<8>(float2 *a) {
    float2 e[4] = {a[0], a[2], a[4], a[6]}, o[4] = {a[1], a[3], a[5], a[7]};
    dft<4>(e);
    dft<4>(o);
    const float h = 0.70710678118654757f;  // sqrt(1/2)
    // o_k * exp(-2 pi i k / 8)
    const float2 o1 = make_float2(h * (o[1].x + o[1].y), h * (o[1].y - o[1].x));
    const float2 o2 = cmi(o[2]);
    const float2 o3 = make_float2(h * (o[3].y - o[3].x), -h * (o[3].x + o[3].y));
    a[0] = cadd(e[0], o[0]);
    a[4] = csub(e[0], o[0]);
    a[1] = cadd(e[1], o1);
    a[5] = csub(e[1], o1);
    a[2] = cadd(e[2], o2);
    a[6] = csub(e[2], o2);
    a[3] = cadd(e[3], o3);
    a[7] = csub(e[3], o3);
}

// v exp(-2 pi i m / N), the quarter and eighth turns without the full product (m is a
// constant once the callers' loops are unrolled)
template <int N>
__device__ __forceinline__ float2 turn(float2 v, int m, const Roots<N> &W) {
    if (m == 0) return v;
    if (4 * m == N) return cmi(v);
    if (2 * m == N) return make_float2(-v.x, -v.y);
    if (4 * m == 3 * N) return make_float2(-v.y, v.x);
    const float h = 0.70710678118654757f;  // sqrt(1/2)
    if (8 * m == N) return make_float2(h * (v.x + v.y), h * (v.y - v.x));
    if (8 * m == 3 * N) return make_float2(h * (v.y - v.x), -h * (v.x + v.y));
    return cmul(v, make_float2(W.c[m], -W.s[m]));
}

// N = N1 N2 point DFT by one mixed-radix split: with n = n1 + N1 n2 and
// k = N2 k1 + k2, b_k = sum_n1 W_N1^(n1 k1) W_N^(n1 k2) sum_n2 W_N2^(n2 k2) a_n:
// N1 inner N2-point DFTs, the twiddles W_N^(n1 k2), N2 outer N1-point DFTs.
template <int N1, int N2>
__device__ __forceinline__ void dft_split(float2 *a) {
    constexpr int N = N1 * N2;
    constexpr Roots<N> W;
    float2 y[N1][N2];
#pragma unroll
    for (int n1 = 0; n1 < N1; ++n1) {
#pragma unroll
        for (int n2 = 0; n2 < N2; ++n2) y[n1][n2] = a[n1 + N1 * n2];
        dft<N2>(y[n1]);
    }
#pragma unroll
    for (int n1 = 1; n1 < N1; ++n1)
#pragma unroll
        for (int k2 = 1; k2 < N2; ++k2) y[n1][k2] = turn<N>(y[n1][k2], n1 * k2 % N, W);
#pragma unroll
    for (int k2 = 0; k2 < N2; ++k2) {
        float2 z[N1];
#pragma unroll
        for (int n1 = 0; n1 < N1; ++n1) z[n1] = y[n1][k2];
        dft<N1>(z);
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) a[N2 * k1 + k2] = z[k1];
    }
}
template <> __device__ __forceinline__ void dft<6>(float2 *a) { dft_split<2, 3>(a); }
template <> __device__ __forceinline__ void dft<9>(float2 *a) { dft_split<3, 3>(a); }
template <> __device__ __forceinline__ void dft<10>(float2 *a) { dft_split<2, 5>(a); }
template <> __device__ __forceinline__ void dft<12>(float2 *a) { dft_split<3, 4>(a); }
template <> __device__ __forceinline__ void dft<14>(float2 *a) { dft_split<2, 7>(a); }
template <> __device__ __forceinline__ void dft<15>(float2 *a) { dft_split<3, 5>(a); }
template <> __device__ __forceinline__ void dft<16>(float2 *a) { dft_split<4, 4>(a); }
template <> __device__ __forceinline__ void dft<18>(float2 *a) { dft_split<2, 9>(a); }
template <> __device__ __forceinline__ void dft<20>(float2 *a) { dft_split<4, 5>(a); }
template <> __device__ __forceinline__ void dft<21>(float2 *a) { dft_split<3, 7>(a); }
template <> __device__ __forceinline__ void dft<22>(float2 *a) { dft_split<2, 11>(a); }
template <> __device__ __forceinline__ void dft<24>(float2 *a) { dft_split<3, 8>(a); }
template <> __device__ __forceinline__ void dft<25>(float2 *a) { dft_split<5, 5>(a); }
template <> __device__ __forceinline__ void dft<26>(float2 *a) { dft_split<2, 13>(a); }
template <> __device__ __forceinline__ void dft<27>(float2 *a) { dft_split<3, 9>(a); }
template <> __device__ __forceinline__ void dft<28>(float2 *a) { dft_split<4, 7>(a); }
template <> __device__ __forceinline__ void dft<30>(float2 *a) { dft_split<2, 15>(a); }
template <> __device__ __forceinline__ void dft<32>(float2 *a) { dft_split<4, 8>(a); }

// Shared-memory index of position p of the thread's vector.  Columns: the NV vectors of a
// position side by side.  Rows: each vector on its own (`at`); between the stages of a
// transform of three or more, one float2 of padding per 16 (operator()), so that a stage's
// stride-r writes spread over the banks.  Between the two stages of a two-stage transform
// both sides are linear: result k of butterfly i of the first stage lies at i * S + k and is
// point q = i of butterfly k of the second, S the first radix (made odd in rows).
template <int NV>
struct ColAddr {
    int v;
    __device__ __forceinline__ int at(int p) const { return p * NV + v; }
    static __device__ __forceinline__ constexpr int at0(int p) { return p * NV; }
    __device__ __forceinline__ int operator()(int p) const { return p * NV + v; }
    static __host__ __device__ __forceinline__ constexpr int between(int r) { return r; }
    static __host__ __device__ int size(int n) { return n * NV; }
    static __device__ __forceinline__ ColAddr of(int v, int) { return ColAddr{v}; }
};
struct RowAddr {
    int base;  // v * pitch(n)
    // at least n + n / 16 + 1, and n / r * (r | 1) of every two-stage plan; odd, so that lanes
    // of different vectors meet no bank conflict (stage_prime)
    static __host__ __device__ int pitch(int n) { return (n + (n >> 3) + 2) | 1; }
    static __device__ __forceinline__ RowAddr of(int v, int n) { return RowAddr{v * pitch(n)}; }
    __device__ __forceinline__ int at(int p) const { return base + p; }
    static __device__ __forceinline__ constexpr int at0(int p) { return p; }
    __device__ __forceinline__ int operator()(int p) const { return base + p + (p >> 4); }
    static __host__ __device__ __forceinline__ constexpr int between(int r) { return r | 1; }
};

// A kernel takes the plans of one group, by the first radix: those to 12 with all plans of
// three and more stages, 13 to 16, and above 16 (as the first of exactly two stages) to 22 and
// to 32.  One switch over all pairs gave every pair the registers of the worst: at 64 a thread
// the image passes reloaded 1000 to 1200 bytes of spills (700 in the first group now, 4 in the
// second), and a pair that joined slowed others (180 points x 256, last pass, 25.6 us, 27.8
// with five more pairs, 24.2 now; 128 points x 16 in 2D 5.8 -> 4.7).
constexpr int group_of(int r0) { return r0 <= 12 ? 0 : r0 <= 16 ? 1 : r0 <= 22 ? 2 : 3; }
constexpr bool big_group(int g) { return g >= 2; }
constexpr int group_most(int g) { return g == 0 ? 12 : g == 1 ? 16 : g == 2 ? 22 : 32; }
#define PFB_FFT_BIG(X) \
    X(17) X(18) X(19) X(20) X(21) X(22) X(23) X(24) X(25) X(26) X(27) X(28) X(29) X(30) X(31) X(32)
#define PFB_FFT_RADICES(X) X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16)

// x_q times the stage's twiddles; the table holds them by q, so that lanes of
// neighbouring j read neighbouring entries
template <int R>
__device__ __forceinline__ void twiddle(float2 *a, const float2 *__restrict__ tw, int ns, int j) {
#pragma unroll
    for (int q = 1; q < R; ++q) a[q] = cmul(a[q], __ldg(tw + j + (q - 1) * ns));
}

// first stage: points through `ld` (position -> value), results to dst; TWO: of two
template <int R, bool TWO, class A, class L>
__device__ __forceinline__ void stage_first(int n, int stream, int T, A ad, L &ld, float2 *__restrict__ dst) {
    const int m = n / R;
    for (int i = stream; i < m; i += T) {
        float2 a[R];
#pragma unroll
        for (int q = 0; q < R; ++q) a[q] = ld(i + q * m);
        dft<R>(a);
        if constexpr (TWO) {
            float2 *d = dst + ad.at(i * A::between(R));
#pragma unroll
            for (int k = 0; k < R; ++k) d[A::at0(k)] = a[k];
        } else {
#pragma unroll
            for (int k = 0; k < R; ++k) dst[ad(i * R + k)] = a[k];
        }
    }
}

template <int R, class A>
__device__ __forceinline__ void stage_mid(int n, int ns, unsigned magic, const float2 *__restrict__ tw, int stream,
                                          int T, A ad, const float2 *__restrict__ src, float2 *__restrict__ dst) {
    const int m = n / R;
    for (int i = stream; i < m; i += T) {
        const int j = ns == 1 ? 0 : i - (int)__umulhi((unsigned)i, magic) * ns;
        float2 a[R];
#pragma unroll
        for (int q = 0; q < R; ++q) a[q] = src[ad(i + q * m)];
        if (ns > 1) twiddle<R>(a, tw, ns, j);
        dft<R>(a);
        const int base = (i - j) * R + j;
#pragma unroll
        for (int k = 0; k < R; ++k) dst[ad(base + k * ns)] = a[k];
    }
}

// last stage (ns = n / r, so j = i): result k of butterfly i is the transform's i + k ns
template <int R, bool TWO, class A, class S>
__device__ __forceinline__ void stage_last(int n, const float2 *__restrict__ tw, int stream, int T, A ad,
                                           const float2 *__restrict__ src, S &st) {
    const int m = n / R;
    const int between = A::between(m);  // of two stages: m is the first radix
    for (int i = stream; i < m; i += T) {
        float2 a[R];
#pragma unroll
        for (int q = 0; q < R; ++q) a[q] = TWO ? src[ad.at(i + q * between)] : src[ad(i + q * m)];
        twiddle<R>(a, tw, m, i);
        dft<R>(a);
#pragma unroll
        for (int k = 0; k < R; ++k) st(i + k * m, a[k]);
    }
}

// A stage whose radix is a prime that no two-stage plan takes, after a radix-1 stage (so
// without twiddles): a thread takes kPrimeOut pairs of outputs (k, r - k) of a butterfly and
// walks the (r - 1) / 2 input pairs.  The table `rt` holds its coefficients in that order as
// (cos, cos, sin, sin) of 2 pi q k / r, the operands of packed FMAs: per input pair and
// output pair one 16-byte load and two FMAs, no index arithmetic (with the roots looked up
// by q k mod r: 36 instructions for 4 output pairs instead of 16; 472 = 8 x 59 points, 31
// coils: 46 -> 21 us a pass).  Primes above kMaxPrime hold (cos, sin) alone: the doubled
// table of 167, 111 KB, misses L1 (y pass of 93 x 111 x 120, 5 coils: 566 us).
constexpr int kPrimeOut = 4;
template <bool DUP, class A>
__device__ __forceinline__ void stage_prime(int n, int R, const float2 *__restrict__ rt, int stream, int T, A ad,
                                            const float2 *__restrict__ src, float2 *__restrict__ dst) {
    const int m = n / R, H = (R - 1) / 2;
    const int ng = (H + kPrimeOut - 1) / kPrimeOut;
    for (int w = stream; w < m * ng; w += T) {
        const int g = w / m, i = w - g * m;
        const float2 x0 = src[ad(i)];
        float2 c[kPrimeOut], s[kPrimeOut], sum = x0;
#pragma unroll
        for (int u = 0; u < kPrimeOut; ++u) {
            c[u] = x0;
            s[u] = make_float2(0.f, 0.f);
        }
        using F = typename std::conditional<DUP, float4, float2>::type;
        const F *r = reinterpret_cast<const F *>(rt) + g * H * kPrimeOut;
#pragma unroll 2
        for (int q = 1; q <= H; ++q, r += kPrimeOut) {
            const float2 a = src[ad(i + q * m)], b = src[ad(i + (R - q) * m)];
            const float2 t = cadd(a, b), d = csub(a, b);
            sum = cadd(sum, t);
#pragma unroll
            for (int u = 0; u < kPrimeOut; ++u) {
                const F f = __ldg(r + u);
                if constexpr (DUP) {
                    c[u] = __ffma2_rn(make_float2(f.x, f.y), t, c[u]);
                    s[u] = __ffma2_rn(make_float2(f.z, f.w), d, s[u]);
                } else {
                    c[u] = cfma(f.x, t, c[u]);
                    s[u] = cfma(f.y, d, s[u]);
                }
            }
        }
        const int base = i * R;
        if (g == 0) dst[ad(base)] = sum;
#pragma unroll
        for (int u = 0; u < kPrimeOut; ++u) {
            const int k = g * kPrimeOut + u + 1;
            if (k > H) break;
            dst[ad(base + k)] = cadd(c[u], cmi(s[u]));
            dst[ad(base + R - k)] = csub(c[u], cmi(s[u]));
        }
    }
}

// A two-stage transform of R0 x R1 points, every length and index a constant.
template <int R0, int R1, class A, class L, class S>
__device__ __forceinline__ void run_two(const float2 *__restrict__ tw, int stream, int T, A ad, float2 *b0, L &ld, S &st) {
    constexpr int SB = A::between(R0);
    for (int i = stream; i < R1; i += T) {
        float2 a[R0];
#pragma unroll
        for (int q = 0; q < R0; ++q) a[q] = ld(i + q * R1);
        dft<R0>(a);
        float2 *d = b0 + ad.at(i * SB);
#pragma unroll
        for (int k = 0; k < R0; ++k) d[A::at0(k)] = a[k];
    }
    __syncthreads();
    for (int i = stream; i < R0; i += T) {
        float2 a[R1];
        const float2 *c = b0 + ad.at(i);
        const float2 *w = tw + i;
#pragma unroll
        for (int q = 0; q < R1; ++q) a[q] = c[A::at0(q * SB)];
#pragma unroll
        for (int q = 1; q < R1; ++q) a[q] = cmul(a[q], __ldg(w + (q - 1) * R0));
        dft<R1>(a);
#pragma unroll
        for (int k = 0; k < R1; ++k) st(i + k * R0, a[k]);
    }
}

// The lengths with constants, in the plans that stage_plan picks: image extents of 64 to 256
// in steps of 16 or 20 at the oversampling factors 1, 1.25 and 1.5 and doubled (Toeplitz
// grids), from 80 points on, where row passes take two stages.  Runtime indices cost the row
// passes as many instructions as the transform itself (256 points: 50 a point and transform
// against about 28).
#define PFB_FFT_TWO(X) \
    X(12, 8) X(10, 10) X(14, 8) X(12, 10) X(16, 8) X(12, 12) X(15, 10) X(16, 10) X(16, 11) X(15, 12) X(16, 12) \
    X(16, 13) X(16, 14) X(16, 15) X(16, 16) X(10, 8) X(14, 10) X(14, 12) X(15, 14) X(15, 15)
#define PFB_FFT_TWO_BIG(X) \
    X(20, 10) X(18, 12) X(20, 11) X(25, 10) X(25, 11) X(18, 16) X(20, 15) X(20, 16) X(22, 16) X(20, 18) X(24, 16) \
    X(20, 20) X(22, 20) X(24, 20) X(32, 16) X(20, 13) X(22, 12) X(18, 15) X(20, 14) X(24, 13) X(22, 15) X(21, 16) \
    X(26, 16) X(28, 16)

// Forward transform of the thread's vector: points through ld(position), results through
// st(frequency, value).  b0 and b1 (b1 only with more than two stages): A::size(n) float2
// of shared memory each, not read by any thread any more when the call begins.
template <int G, class A, class L, class S>
__device__ __forceinline__ void run(const FftAxis &fa, int stream, int T, A ad, float2 *b0, float2 *b1, L &ld, S &st) {
    const int n = fa.n, nst = fa.nst;
    if (G > 0 || nst == 2) {
        switch (fa.radix[0] * 32 + fa.radix[1]) {
#define X(R0, R1) \
    case R0 * 32 + R1: \
        if constexpr (group_of(R0) == G) run_two<R0, R1>(fa.tw + fa.twoff[1], stream, T, ad, b0, ld, st); \
        return;
            PFB_FFT_TWO(X) PFB_FFT_TWO_BIG(X)
#undef X
            default: break;
        }
        switch (fa.radix[0]) {
#define X(R) \
    case R: \
        if constexpr (group_of(R) == G) stage_first<R, true>(n, stream, T, ad, ld, b0); \
        break;
            PFB_FFT_RADICES(X) PFB_FFT_BIG(X)
#undef X
            default: break;
        }
        __syncthreads();
        const float2 *tw = fa.tw + fa.twoff[1];
        switch (fa.radix[1]) {
#define X(R) \
    case R: \
        if constexpr (R <= group_most(G)) stage_last<R, true>(n, tw, stream, T, ad, b0, st); \
        break;
            PFB_FFT_RADICES(X) PFB_FFT_BIG(X)
#undef X
            default: break;
        }
        return;
    }
    if constexpr (G == 0) {
        switch (fa.radix[0]) {
#define X(R) \
    case R: stage_first<R, false>(n, stream, T, ad, ld, b0); break;
            PFB_FFT_RADICES(X)
#undef X
            default: break;
        }
        __syncthreads();
        float2 *src = b0, *dst = b1;
        for (int s = 1; s + 1 < nst; ++s) {
            const int ns = fa.ns[s];
            const unsigned mg = fa.magic[s];
            const float2 *tw = fa.tw + fa.twoff[s];
            switch (fa.radix[s]) {
#define X(R) \
    case R: stage_mid<R>(n, ns, mg, tw, stream, T, ad, src, dst); break;
                PFB_FFT_RADICES(X)
#undef X
                default: {
                    // lanes along the vectors in row passes too: the lanes of a warp then
                    // share a group of outputs and its coefficients
                    const int V = blockDim.x / T, pv = threadIdx.x % V;
                    if (fa.radix[s] <= kMaxPrime)
                        stage_prime<true>(n, fa.radix[s], fa.tw + fa.rootoff[s], threadIdx.x / V, T, A::of(pv, n), src,
                                          dst);
                    else
                        stage_prime<false>(n, fa.radix[s], fa.tw + fa.rootoff[s], threadIdx.x / V, T, A::of(pv, n), src,
                                           dst);
                    break;
                }
            }
            __syncthreads();
            float2 *t = src;
            src = dst;
            dst = t;
        }
        const float2 *tw = fa.tw + fa.twoff[nst - 1];
        switch (fa.radix[nst - 1]) {
#define X(R) \
    case R: stage_last<R, false>(n, tw, stream, T, ad, src, st); break;
            PFB_FFT_RADICES(X)
#undef X
            default: break;
        }
    }
}

}  // namespace fft
}  // namespace pfb
