// The passes of the fused FFT (pfb_fft.cu): their arguments and launch shapes.
#pragma once

#include "pfb_fft.cuh"

namespace pfb {
namespace fft {

constexpr int kMaxN = 1024;        // longest axis handled (else the library FFT)
constexpr int kMaxThreads = 256;   // threads per CTA
// CTAs per SM that bound the registers: 64 a thread, or 128 with a radix above 16
constexpr int min_blocks(bool big) { return big ? 2 : 4; }
inline int plan_group(const FftAxis &fa) { return fa.nst == 2 ? group_of(fa.radix[0]) : 0; }

// Division of 0 <= e < 2^31 by a divisor known at the launch, as a multiply-high and a
// shift.  A CTA of the direct passes lives for one tile, 16 points or so a thread: a handful
// of integer divisions for its coordinates cost as much as the transform (256 points: 55
// instructions a point with them).
struct Div {
    unsigned m = 0;
    int sh = 0, d = 1;
    Div() = default;
    explicit Div(int v) : d(v < 1 ? 1 : v) {
        if (d > 1) {
            int L = 1;
            while ((1ll << L) < d) ++L;
            m = (unsigned)((1ull << (31 + L)) / (unsigned)d + 1);
            sh = L - 1;
        }
    }
#ifdef __CUDACC__
    __device__ __forceinline__ int operator()(int e) const { return d == 1 ? e : (int)(__umulhi((unsigned)e, m) >> sh); }
    // e / d, and e mod d in r
    __device__ __forceinline__ int split(int e, int &r) const {
        const int q = (*this)(e);
        r = e - q * d;
        return q;
    }
#endif
};

// column passes: image -> buffer, buffer -> buffer forward / inverse, buffer -> image
enum { kImageIn = 0, kForward = 1, kInverse = 2, kImageOut = 3, kRowForward = 4, kRowInverse = 5 };

// Transform along an outer axis (y or z).  Forward passes read lin = N elements placed at
// FFT positions (i - N/2) mod n and write all n; inverse passes read all n and write
// lout = N, element o from FFT position (o - N/2) mod n.  Strides are in elements (along
// the axis below 2^31); for the image side they are the image strides.
struct ColPass {
    FftAxis fa;
    int lin, lout, nax;
    int X, nmid, nplanes;
    int64_t in_plane, in_mid, in_ax;
    int64_t out_plane, out_mid, out_ax;
    const float2 *src;
    float2 *dst;
    Chan ch;
    int C;
    int64_t nvol;
    const float *apod_ax, *apod_mid, *apod_x;
    const float2 *Cl;
    float factor;
    int accumulate;
    int *err;  // device flag of the plan (TMA form: a wait that gave up)
    int nsm;   // SMs of the device (TMA form: persistent grid)
    int T;     // set by the launch: threads per vector, and the divisors of a CTA's coordinates
    Div dx, dmid, dnch, dk, db, dc;
};

// Transform along x (see the kernels for the layouts)
struct RowPass {
    FftAxis fa;
    int N0;
    int64_t nvec;
    int nch, nos1, nos2;
    int64_t gvol;
    const float2 *src;
    float2 *dst;
    int *err;  // as ColPass
    int nsm;
    // set by the launch
    int V, T, buf;                    // vectors per CTA, threads per vector, float2 per shared buffer
    int cpt, nchunk, kpt, nyb, cp;    // channels per tile, chunks, rows per tile, tiles along ky, output pitch
    Div dt, dchunk, dyb, dz, dcpt, dunit;  // dunit: store units of a full tile
};

// The Gram's middle pass (pfb_fft_gram.cu): rows of the grid, N0 of n points held, in place
struct GramRows {
    FftAxis fa;
    int N0, rows;             // points held per row; rows of the grid (n1 x n2)
    int K, lowrank, batch, nseg;
    int64_t gvol;             // points of the kernel per segment (and plane)
    const float2 *kern;       // K x K matrices per point, or K planes; a leading segment axis
    float2 *grid;             // [segment][batch][K][row][N0]
    int V, T, nbv, nbg;       // set by the launch: vectors and threads, batch items per CTA, groups
    Div dt, dbg, dk, drow;
};
int launch_gram_rows(const GramRows &P, cudaStream_t s);

// TMA forms (pfb_fft_tma.cu): 1 if launched, 0 to take the direct form, or an error
int launch_col_tma(const ColPass &P, int pass, cudaStream_t s);
int launch_row_tma(const RowPass &P, bool inv, cudaStream_t s);
int launch_col(const ColPass &P, int mode, cudaStream_t s);
// one instantiation per file (pfb_fft_cols_*.cu, pfb_fft_gram*.cu), so that they compile side by side
template <int MODE, int G>
int launch_col_mode(const ColPass &P, cudaStream_t s);
template <int G>
int launch_gram_rows_t(const GramRows &P, cudaStream_t s);
int launch_row(const RowPass &P, bool inv, cudaStream_t s);

// Threads per vector of a CTA with nv vectors and `smem` bytes, `blocks` of them in the
// launch: the count (64 to kMaxThreads threads; from 32 for a vector alone, the Gram rows of a
// single image: 96^3 on 192^3 133 -> 95 us) that leaves the fewest thread slots idle
// over the stages' rounds, a butterfly of radix r costing about r + 2, as long as the CTAs
// that share an SM have kFullWarps warps.  With fewer (long vectors, whose CTAs shared
// memory limits to a few per SM, or few CTAs) the latency of a warp counts instead of its
// slots, and more threads in fewer rounds are the faster.  By the idle
// slots alone 624 points ran in CTAs of 64 threads, 10 warps an SM, at 15 % issue slots
// (2D, 12 channels, a forward and an adjoint, us: 624 points 69 + 134, now 65 + 102; 640
// points 77 + 125, now 71 + 100; 936 points 258 + 395, now 174 + 248; over 12086 calls of
// 16 to 1024 points 1.03 times as fast, 16 warps 1.04 but 10 % slower around 400 points).
// With a prime stage, whose items are long, the count within a quarter of that which takes
// them in the fewest rounds (118 = 2 x 59 points, y pass, 34 us with two rounds and 15 us
// with one); not for those above kMaxPrime, whose passes are bound by throughput (167
// points: 454 us by the first rule).  At least `least` (row passes: lanes along the row,
// whole 128-byte segments).
constexpr int kFullWarps = 12;
inline int streams(const FftAxis &fa, int nv, size_t smem, int64_t blocks, int least = 1) {
    // CTAs per SM: shared memory (1 KB each is the system's), and the launch's share of the 148
    const int fit = (int)std::min<int64_t>(227 * 1024 / (int64_t)(smem + 1024), (blocks + 147) / 148);
    const int regs = min_blocks(big_group(plan_group(fa))) * kMaxThreads / 32;  // warps that the registers hold
    const int t0 = std::max((nv == 1 ? 32 : 64) / nv, std::max(least, 1));
    int best = 0, rounds = 0, width = 0;
    double low = 1e300, cost = 1e300, steps = 0;
    bool has_prime = false;
    for (int pass = 0; pass < 2; ++pass) {
        for (int t = t0; t * nv <= kMaxThreads || best == 0; ++t) {
            double n = 0;  // steps of a thread, one after the other
            int pr = 0;
            for (int s = 0; s < fa.nst; ++s) {
                const int r = fa.radix[s], m = fa.n / r;
                if (r > 16 && s > 0 && s + 1 < fa.nst) {  // pairs of outputs in groups of 4, r / 2 steps each
                    const int w = m * (((r - 1) / 2 + 3) / 4);
                    n += (double)((w + t - 1) / t) * (2.0 * r);
                    pr += (w + t - 1) / t;
                    has_prime = has_prime || r <= kMaxPrime;
                } else {
                    n += (double)((m + t - 1) / t) * (r + 2.0);
                }
            }
            const int warps = (t * nv + 31) / 32, ctas = std::max(1, std::min(fit, regs / warps));
            const double c = n * std::max((double)warps, (double)kFullWarps / ctas);
            // on a tie the fewer steps, and more threads only within the same warps
            const bool tie = n < steps || (n == steps && warps == width);
            if (pass == 0 ? c < low || (c == low && tie)
                          : c <= 1.25 * low && (rounds == 0 || pr < rounds || (pr == rounds && (c < cost || (c == cost && tie))))) {
                if (pass == 0) low = c;
                else rounds = pr;
                best = t, cost = c, steps = n, width = warps;
            }
        }
        if (!has_prime) break;
    }
    return best;
}

// 8 instead of 16 columns per CTA: above 128 points (more CTAs in flight per SM: 180 points,
// y pass of 120^3 x 16 at osf 1.5, 194 -> 169 us; 128 points 171 against 185 us the other
// way), and for passes with too few tiles to fill the chip
inline bool narrow_tiles(int n, int64_t tiles) { return n > 128 || tiles < 296; }

}  // namespace fft
}  // namespace pfb
