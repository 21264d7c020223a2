// Fused, pruned FFT of the channel-interleaved NUFFT pipeline (2D and 3D).
//
// The reference's glue around the library FFT (src/pyfourier/_subroutines/_fft.py:72-79
// via _nufft/_nufft.py:218-287) is pad -> centred FFT -> (interpolate) and
// (spread) -> centred inverse FFT -> crop, with deapodisation (_apod.py:16-46) and
// the B0 spatial factors applied on the image side.  Here the multi-dimensional
// transform is run axis by axis as batched 1D transforms in registers and shared memory
// (pfb_fft.cuh), and the passes are pruned and fused with their neighbours:
//
//   forward 3D: image --(z pass: deapodise, C_l, zero-pad, FFT)--> T1[plane][kz][y][x]
//               --(y pass)--> T2[plane][kz][ky][x] --(x pass)--> interleaved grid
//   adjoint 3D: planar grid --(x pass: IFFT, crop x)--> T1[plane][kz][ky][x]
//               --(y pass: crop y)--> T2[plane][kz][y][x]
//               --(z pass: crop z, sum_l conj(C_l), deapodise)--> image
//
// (2D drops the z pass.)  Rows and columns that are all zero are never read or
// written, so a forward transform of an N^3 image onto an n^3 grid moves about
// N^3 + 2 n N^2 + 2 n^2 N + n^3 elements per plane instead of the 2 n^3 per pass
// of an unpruned transform, and the pad, crop and channel transpose cost nothing
// extra.  The passes' kernels: pfb_fft_cols.cuh, pfb_fft_rows.cu, pfb_fft_tma.cu.
#include <cmath>
#include <vector>

#include "pfb_fft_passes.cuh"

namespace pfb {
using namespace fft;
namespace fft {

template <int MODE>
static int launch_col_direct(const ColPass &P, cudaStream_t s) {
    switch (plan_group(P.fa)) {
        case 0: return launch_col_mode<MODE, 0>(P, s);
        case 1: return launch_col_mode<MODE, 1>(P, s);
        case 2: return launch_col_mode<MODE, 2>(P, s);
        default: return launch_col_mode<MODE, 3>(P, s);
    }
}

int launch_col(const ColPass &P, int mode, cudaStream_t s) {
    if (P.nplanes == 0 || P.nmid == 0 || P.X == 0) return PFB_OK;
    const int st = launch_col_tma(P, mode, s);
    if (st) return st == 1 ? PFB_OK : st;
    switch (mode) {
        case kImageIn: return launch_col_direct<kImageIn>(P, s);
        case kForward: return launch_col_direct<kForward>(P, s);
        case kInverse: return launch_col_direct<kInverse>(P, s);
        default: return launch_col_direct<kImageOut>(P, s);
    }
}

int launch_gram_rows(const GramRows &P, cudaStream_t s) {
    if (P.batch == 0 || P.rows == 0) return PFB_OK;
    switch (plan_group(P.fa)) {
        case 0: return launch_gram_rows_t<0>(P, s);
        case 1: return launch_gram_rows_t<1>(P, s);
        case 2: return launch_gram_rows_t<2>(P, s);
        default: return launch_gram_rows_t<3>(P, s);
    }
}

}  // namespace fft
namespace {

// the radices that exist
bool is_radix(int r) { return r >= 2 && r <= 32; }

// Non-increasing factors of n in 2..16, as few as possible and then as even as possible
// (the least sum), appended to f.  False if n has another prime factor.
bool split_smooth(int n, std::vector<int> &f) {
    if (n == 1) return true;
    std::vector<int> cur, best;
    auto sum = [](const std::vector<int> &v) {
        int t = 0;
        for (int x : v) t += x;
        return t;
    };
    auto rec = [&](auto &&self, int m, int most) -> void {
        if (m == 1) {
            if (best.empty() || cur.size() < best.size() || (cur.size() == best.size() && sum(cur) < sum(best)))
                best = cur;
            return;
        }
        if (!best.empty() && cur.size() >= best.size()) return;
        for (int r = std::min(most, m); r >= 2; --r)
            if (m % r == 0) {
                cur.push_back(r);
                self(self, m / r, r);
                cur.pop_back();
            }
    };
    rec(rec, n, 16);
    f.insert(f.end(), best.begin(), best.end());
    return !best.empty();
}

// The stages of an n-point transform: two stages up to 16 where they exist, then two up to
// 32 (in row passes, whose lanes run along the n / r butterflies of the first stage, a
// length that also splits into three stages up to 16 only where that leaves at least 8:
// 125 points as 25 x 5 214 us, as 5 x 5 x 5 158 us for 100^3 x 12), then three or more: the
// largest radix first and the next largest last.  A prime above 13 that no pair takes is
// the middle stage of three; the first and the last, which read and write global memory,
// then hold the rest of the length (a radix-1 stage copies).  False when there is no such plan.
bool stage_plan(int n, bool rows, std::vector<int> &rad) {
    if (n < 1 || n > kMaxN) return false;
    std::vector<int> primes, f;
    int m = n;
    for (int p = 17; p <= kMaxPrime3; ++p)
        while (m % p == 0) {
            bool prime = true;
            for (int d = 2; d * d <= p; ++d) prime = prime && p % d != 0;
            if (!prime) break;
            primes.push_back(p);
            m /= p;
        }
    if (!split_smooth(m, f)) return false;
    if (!primes.empty() || f.size() > 2) {
        int big = 0;
        for (int r = 32; r >= 17; --r)  // the more even split last
            if (n % r == 0 && n / r <= r && is_radix(r) && (n / r == 1 || is_radix(n / r)) &&
                (!rows || n / r >= 8 || !primes.empty()))
                big = r;
        if (big) {
            rad = {big, n / big};
            return true;
        }
    }
    if (!primes.empty()) {
        if (primes.size() > 1 || f.size() > 1) return false;
        rad = {1, primes[0], f.empty() ? 1 : f[0]};
        return true;
    }
    rad = {f.empty() ? 1 : f[0]};
    for (size_t i = 2; i < f.size(); ++i) rad.push_back(f[i]);
    rad.push_back(f.size() > 1 ? f[1] : 1);
    return (int)rad.size() <= kFftMaxStages;
}

// the pair has a form with constants (run_two)
constexpr bool constant_pair(int r0, int r1) {
#define X(R0, R1) if (r0 == R0 && r1 == R1) return true;
    PFB_FFT_TWO(X) PFB_FFT_TWO_BIG(X)
#undef X
    return false;
}

// The prime of a plan's prime stage, 0 without one.
int prime_stage(const std::vector<int> &rad) { return rad.size() == 3 && rad[1] > 16 ? rad[1] : 0; }

constexpr double kPi = 3.14159265358979323846;

unsigned magic_of(int d) { return d > 1 ? (unsigned)(0xFFFFFFFFull / (unsigned long long)d + 1ull) : 0u; }

// Appends the axis's twiddles (by q, see twiddle()) and the roots of its prime stages to
// tw: offsets are relative to *base, the axis's first entry.
bool make_axis(int n, bool rows, FftAxis *fa, std::vector<float2> &tw, size_t *base) {
    *fa = FftAxis{};
    std::vector<int> rad;
    if (!stage_plan(n, rows, rad)) return false;
    fa->n = n;
    fa->nst = (int)rad.size();
    if (tw.size() % 2) tw.push_back(make_float2(0.f, 0.f));
    *base = tw.size();
    auto root = [&](double num, double den) {
        const double ang = -2.0 * kPi * num / den;
        tw.push_back(make_float2((float)std::cos(ang), (float)std::sin(ang)));
    };
    int ns = 1;
    for (int s = 0; s < fa->nst; ++s) {
        const int r = rad[s];
        fa->radix[s] = r;
        fa->ns[s] = ns;
        fa->twoff[s] = (int)(tw.size() - *base);
        fa->magic[s] = magic_of(ns);
        for (int q = 1; q < r; ++q)
            for (int j = 0; j < ns; ++j) root((double)j * q, (double)ns * r);
        if (s > 0 && s + 1 < fa->nst && r > 16) {  // coefficients of a prime stage, see stage_prime
            if (tw.size() % 2) tw.push_back(make_float2(0.f, 0.f));  // 16-byte entries
            fa->rootoff[s] = (int)(tw.size() - *base);
            const int H = (r - 1) / 2;
            for (int g = 0; g * kPrimeOut < H; ++g)
                for (int q = 1; q <= H; ++q)
                    for (int u = 0; u < kPrimeOut; ++u) {
                        const int k = std::min(g * kPrimeOut + u + 1, H);
                        const double ang = 2.0 * kPi * (q * k % r) / r;
                        const float c = (float)std::cos(ang), d = (float)std::sin(ang);
                        if (r <= kMaxPrime) {
                            tw.push_back(make_float2(c, c));
                            tw.push_back(make_float2(d, d));
                        } else {
                            tw.push_back(make_float2(c, d));
                        }
                    }
        }
        ns *= r;
    }
    if (rows && fa->nst == 2) {  // see gram_two
        fa->swapoff = (int)(tw.size() - *base);
        for (int q = 1; q < rad[0]; ++q)
            for (int j = 0; j < rad[1]; ++j) root((double)j * q, (double)n);
    }
    return true;
}

}  // namespace

// Which grids the passes take: those where they are the faster, of 12000 calls on grids of 16
// to 1024 points an axis in 2D and 3D (NUFFTs of few samples, so that the transform is most of
// the call, and Gram operators), timed on the library's transform and here.  Figures: us,
// library / here; 2D with 12 channels, 3D with 4, 64 points on the other axes, where not said.
//
// - Two stages, to 1024 points: taken (640^2 forward, with the pad and transpose that the
//   library needs, 121 / 71, adjoint 110 / 100; of all lengths the slowest are thin grids
//   with a long z axis: 425 points, forward 174 / 134, adjoint 150 / 169).
// - Three stages and more: their second buffer leaves few CTAs to an SM.  Taken to 768 points
//   (735^2 194 / 117 and 189 / 146; 1000^2 239 / 198 but 227 / 291).
// - A prime stage, O(r^2): to 512 points (561^2 101 / 102 and 100 / 135) for primes to 64 (2D
//   1.5 times as fast, 3D 1.1 to 1.4); for primes to kMaxPrime where the stage is the axis or
//   half of it (254^2 87 / 69 and 89 / 73; 508^2 139 / 204 and 141 / 220), in 3D the whole
//   axis only beside axes that make up for it (83 points in y 72 / 73 and 71 / 81; 89 beside
//   96 x 96, 6 channels, 199 / 120 and 172 / 138); for primes to kMaxPrime3 on such an axis, y
//   or z, that is at least 1.5 times its image, so that the passes skip a third of it (111 of
//   167 points in y, 150 x 150, 16 channels, 2129 / 1514 and 1956 / 1772; 166 of 167 points
//   2237 / 2268 and 2148 / 2508; 115 of 173, 128 x 128, 1086 / 989 and 894 / 1113).
//   Two axes of a 3D grid that are such primes: not (16 planes of 61^3 454 / 509, 107^3 2908 /
//   3538; with one, 96 x 96 x 107, 1426 / 1290).
// - A Gram whose grid is the image is transformed in place by the library, without pad and
//   crop: taken in 2D with at most 5 coefficients, at 96 to 400 points in two stages with
//   constants (256^2 x 4, 12 images 71 / 53, 256 images 896 / 853; elementwise 31 / 24) and to
//   288 points without, where the last radix is not small (1.05 to 1.3 times as fast by the
//   number of images and coefficients; single images of 3 MB from 0.85 to 1.3; 27 x 9 points
//   0.8, 17 x 17 0.9).  With 8 coefficients 256^2 takes 146 / 187 (128 images 1065 / 1693); in 3D 64^3 29 / 40,
//   64 of them 368 / 395.
// - A low-rank Gram holds all K planes of a row twice in shared memory: taken to 64 KB (8
//   planes of 440 points 491 / 417, of 1024 points 1538 / 2343).
static bool fused_takes(int ndim, const int *n, const int *nos, const GramRoute *gram) {
    if (ndim < 2) return false;
    bool dense = gram && gram->nseg == 1;
    for (int a = 0; a < ndim; ++a) dense = dense && n[a] == nos[a];
    if (dense && (ndim != 2 || gram->lowrank > 5)) return false;
    int bare = 0;
    for (int a = 0; a < ndim; ++a) {
        std::vector<int> rad;
        if (!stage_plan(nos[a], a == 0, rad)) return false;
        const int len = nos[a], p = prime_stage(rad);
        if (dense) {
            if (rad.size() != 2 || len < 96) return false;
            if (!(constant_pair(rad[0], rad[1]) && len <= 400) && !(len <= 288 && (rad[0] <= 16 || rad[1] >= 10)))
                return false;
        } else if (rad.size() > 2 && !p) {
            if (len > 768) return false;
        } else if (p) {
            if (len > 512) return false;
            if (p > 48 && p == len) ++bare;
            int64_t other = 1;
            for (int b = 0; b < ndim; ++b) other *= b == a ? 1 : nos[b];
            if (p > 64) {
                if (p > kMaxPrime ? ndim == 2 || p != len || a == 0 || 2 * (int64_t)len < 3 * (int64_t)n[a] : len > 2 * p)
                    return false;
                if (ndim == 3 && p == len && other < 96 * 96) return false;
            }
        }
    }
    if (ndim == 3 && bare >= 2) return false;
    // two buffers of K rows
    return !gram || 2 * gram->lowrank * RowAddr::pitch(nos[0]) * (int)sizeof(float2) <= 64 * 1024;
}

int fft_route(int ndim, const int *n, const int *nos, const GramRoute *gram) { return fused_takes(ndim, n, nos, gram) ? 1 : 0; }

int fft_axes(int ndim, const int *n, const int *nos, const GramRoute *gram, FftAxis *ax, float2 **d_tw) {
    *d_tw = nullptr;
    if (!fused_takes(ndim, n, nos, gram)) return 0;
    std::vector<float2> tw;
    size_t base[3] = {0, 0, 0};
    for (int a = 0; a < ndim; ++a)
        if (!make_axis(nos[a], a == 0, &ax[a], tw, &base[a])) return 0;
    if (tw.empty()) tw.push_back(make_float2(1.f, 0.f));
    if (pool_alloc(reinterpret_cast<void **>(d_tw), tw.size() * sizeof(float2)) != PFB_OK) return 0;
    if (upload_table(*d_tw, tw.data(), tw.size() * sizeof(float2)) != PFB_OK) {
        pool_free(*d_tw, 0);
        *d_tw = nullptr;
        return 0;
    }
    for (int a = 0; a < ndim; ++a) ax[a].tw = *d_tw + base[a];
    return 1;
}

int fft_fused_ready(pfb_plan *p) {
    std::lock_guard<std::mutex> lk(p->fft_mu);
    if (p->fft_fused >= 0) return p->fft_fused;
    p->fft_fused = 0;
    if (!fft_axes(p->g.ndim, p->g.n, p->g.nos, nullptr, p->fft_ax, &p->d_fft_tw)) return 0;
    // the TMA passes' flag and persistent grid (optional: without them the direct passes run)
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&p->fft_nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        p->fft_nsm = 0;
    if (pool_alloc(reinterpret_cast<void **>(&p->d_fft_err), sizeof(int)) != PFB_OK) {
        p->d_fft_err = nullptr;
    } else if (clear_table(p->d_fft_err, sizeof(int)) != PFB_OK) {
        pool_free(p->d_fft_err, 0);
        p->d_fft_err = nullptr;
    }
    p->fft_fused = 1;
    return 1;
}

void fft_fused_free(pfb_plan *p) {
    std::lock_guard<std::mutex> lk(p->fft_mu);
    // called with the device synchronised (plan destruction)
    pool_free(p->d_fft_tw, 0);
    p->d_fft_tw = nullptr;
    pool_free(p->d_fft_err, 0);
    p->d_fft_err = nullptr;
    p->fft_fused = -1;
}

int fft_fused_fwd(pfb_plan *p, int pass, const Chan &c, int C, const float2 *img, const float *const *apod,
                  const float2 *Cl, float factor, float2 *gridp, float2 *gridi, cudaStream_t s) {
    const Geom &g = p->g;
    const int D = g.ndim;
    const int P = c.ngrp * c.nch;
    const int64_t N0 = g.n[0], N1 = g.n[1], n1 = g.nos[1], n2 = g.nos[2];
    if (pass == 0) {  // image -> first intermediate: z pass (3D) into gridi, or y pass (2D) into gridp
        ColPass Q{};
        Q.err = p->d_fft_err;
        Q.nsm = p->fft_nsm;
        Q.X = (int)N0;
        Q.nplanes = P;
        Q.src = img;
        Q.ch = c;
        Q.C = C;
        Q.nvol = g.nvol;
        Q.Cl = Cl;
        Q.factor = factor;
        Q.apod_x = apod[0];
        if (D == 3) {
            Q.fa = p->fft_ax[2];
            Q.lin = Q.nax = g.n[2];
            Q.lout = (int)n2;
            Q.nmid = (int)N1;
            Q.in_mid = N0;
            Q.in_ax = N1 * N0;
            Q.out_plane = n2 * N1 * N0;
            Q.out_mid = N0;
            Q.out_ax = N1 * N0;
            Q.apod_ax = apod[2];
            Q.apod_mid = apod[1];
            Q.dst = gridi;
        } else {
            Q.fa = p->fft_ax[1];
            Q.lin = Q.nax = (int)N1;
            Q.lout = (int)n1;
            Q.nmid = 1;
            Q.in_mid = 0;
            Q.in_ax = N0;
            Q.out_plane = n1 * N0;
            Q.out_mid = 0;
            Q.out_ax = N0;
            Q.apod_ax = apod[1];
            Q.apod_mid = nullptr;
            Q.dst = gridp;
        }
        return launch_col(Q, kImageIn, s);
    }
    if (pass == 1) {  // 3D: y pass, gridi -> gridp
        if (D != 3) return PFB_OK;
        ColPass Q{};
        Q.err = p->d_fft_err;
        Q.nsm = p->fft_nsm;
        Q.fa = p->fft_ax[1];
        Q.lin = Q.nax = (int)N1;
        Q.lout = (int)n1;
        Q.X = (int)N0;
        Q.nmid = (int)n2;
        Q.nplanes = P;
        Q.in_plane = n2 * N1 * N0;
        Q.in_mid = N1 * N0;
        Q.in_ax = N0;
        Q.out_plane = n2 * n1 * N0;
        Q.out_mid = n1 * N0;
        Q.out_ax = N0;
        Q.src = gridi;
        Q.dst = gridp;
        return launch_col(Q, kForward, s);
    }
    // x pass: gridp rows -> interleaved grid
    RowPass R{};
    R.err = p->d_fft_err;
    R.nsm = p->fft_nsm;
    R.fa = p->fft_ax[0];
    R.N0 = (int)N0;
    R.nch = c.nch;
    R.nos1 = (int)n1;
    R.nos2 = D == 3 ? (int)n2 : 1;
    R.nvec = (int64_t)c.ngrp * R.nos2 * R.nos1 * c.nch;
    R.gvol = g.gvol;
    R.src = gridp;
    R.dst = gridi;
    return launch_row(R, false, s);
}

int fft_fused_adj(pfb_plan *p, int pass, const Chan &c, int C, float2 *img, const float *const *apod,
                  const float2 *Cl, float factor, bool accumulate, float2 *gridp, float2 *gridi, cudaStream_t s) {
    const Geom &g = p->g;
    const int D = g.ndim;
    const int P = c.ngrp * c.nch;
    const int64_t N0 = g.n[0], N1 = g.n[1], n1 = g.nos[1], n2 = g.nos[2];
    if (pass == 0) {
        // x pass: planar grid rows -> gridi, cropped to N0
        RowPass R{};
        R.err = p->d_fft_err;
        R.nsm = p->fft_nsm;
        R.fa = p->fft_ax[0];
        R.N0 = (int)N0;
        R.nos1 = (int)n1;
        R.nos2 = D == 3 ? (int)n2 : 1;
        R.nvec = (int64_t)P * R.nos2 * R.nos1;
        R.src = gridp;
        R.dst = gridi;
        int st = launch_row(R, true, s);
        if (st || D != 3) return st;
        // 3D: y pass, gridi -> gridp, cropped to N1
        ColPass Q{};
        Q.err = p->d_fft_err;
        Q.nsm = p->fft_nsm;
        Q.fa = p->fft_ax[1];
        Q.lin = (int)n1;
        Q.lout = Q.nax = (int)N1;
        Q.X = (int)N0;
        Q.nmid = (int)n2;
        Q.nplanes = P;
        Q.in_plane = n2 * n1 * N0;
        Q.in_mid = n1 * N0;
        Q.in_ax = N0;
        Q.out_plane = n2 * N1 * N0;
        Q.out_mid = N1 * N0;
        Q.out_ax = N0;
        Q.src = gridi;
        Q.dst = gridp;
        return launch_col(Q, kInverse, s);
    }
    // last pass -> image: z pass (3D, from gridp) or y pass (2D, from gridi)
    ColPass Q{};
    Q.err = p->d_fft_err;
    Q.nsm = p->fft_nsm;
    Q.X = (int)N0;
    Q.nplanes = c.B * C;
    Q.ch = c;
    Q.C = C;
    Q.nvol = g.nvol;
    Q.Cl = Cl;
    Q.factor = factor;
    Q.accumulate = accumulate ? 1 : 0;
    Q.apod_x = apod[0];
    Q.dst = img;
    if (D == 3) {
        Q.fa = p->fft_ax[2];
        Q.lin = (int)n2;
        Q.lout = Q.nax = g.n[2];
        Q.nmid = (int)N1;
        Q.in_plane = n2 * N1 * N0;
        Q.in_mid = N0;
        Q.in_ax = N1 * N0;
        Q.out_mid = N0;
        Q.out_ax = N1 * N0;
        Q.apod_ax = apod[2];
        Q.apod_mid = apod[1];
        Q.src = gridp;
    } else {
        Q.fa = p->fft_ax[1];
        Q.lin = (int)n1;
        Q.lout = Q.nax = (int)N1;
        Q.nmid = 1;
        Q.in_plane = n1 * N0;
        Q.in_mid = 0;
        Q.in_ax = N0;
        Q.out_mid = 0;
        Q.out_ax = N0;
        Q.apod_ax = apod[1];
        Q.apod_mid = nullptr;
        Q.src = gridi;
    }
    return launch_col(Q, kImageOut, s);
}

namespace {
// the Gram's grids: [plane][n2][N1][N0] after the z pass (3D) and [plane][n2][n1][N0]
// before the rows; a dense Gram (N = n on every axis, one segment) works in the output
bool gram_dense(const GramFused &g) {
    bool d = g.nseg == 1;
    for (int a = 0; a < g.ndim; ++a) d = d && g.n[a] == g.nos[a];
    return d;
}
size_t up256(size_t x) { return (x + 255) / 256 * 256; }
}  // namespace

size_t gram_fused_workspace(const GramFused &g, int64_t batch) {
    if (gram_dense(g)) return 256;
    const int64_t P = (int64_t)g.nseg * batch * g.K, n2 = g.ndim == 3 ? g.nos[2] : 1;
    const size_t rows = up256((size_t)(P * n2 * g.nos[1] * g.n[0]) * sizeof(float2));
    return rows + (g.ndim == 3 ? up256((size_t)(P * n2 * g.n[1] * g.n[0]) * sizeof(float2)) : 0);
}

int gram_fused_apply(const GramFused &g, const float2 *image, float2 *out, int64_t batch, const float2 *Cl, void *ws,
                     cudaStream_t s) {
    const int64_t bk = batch * g.K, P = g.nseg * bk;
    const int64_t N0 = g.n[0], N1 = g.n[1], n1 = g.nos[1], n2 = g.ndim == 3 ? g.nos[2] : 1;
    if (P >= (1LL << 31) || n1 * n2 >= (1LL << 31)) return fail(PFB_ERR_UNSUPPORTED, "too many planes for the Gram");
    const bool dense = gram_dense(g);
    float2 *rows = dense ? out : static_cast<float2 *>(ws);
    float2 *zgrid = dense ? out : reinterpret_cast<float2 *>(static_cast<char *>(ws) +
                                                             up256((size_t)(P * n2 * n1 * N0) * sizeof(float2)));
    // images and segments as channels of one group; no fftshift rotation (the embedding
    // sits at the origin)
    ColPass Q{};
    Q.X = (int)N0;
    Q.ch.nch = (int)P;
    Q.ch.ngrp = 1;
    Q.ch.B = (int)bk;
    Q.ch.L = g.nseg;
    Q.C = 1;
    Q.nvol = g.nvol;
    Q.Cl = Cl;
    Q.factor = 1.f;
    // the outermost axis, on the image side
    const int za = g.ndim - 1;
    Q.fa = g.ax[za];
    Q.lin = Q.lout = g.n[za];
    Q.nmid = g.ndim == 3 ? (int)N1 : 1;
    ColPass F = Q, I = Q;
    const int64_t zmid = g.ndim == 3 ? N0 : 0, zax = g.ndim == 3 ? N1 * N0 : N0, zplane = g.nos[za] * zax;
    F.nplanes = (int)P;
    F.in_mid = F.out_mid = I.in_mid = I.out_mid = zmid;
    F.in_ax = F.out_ax = I.in_ax = I.out_ax = zax;
    F.out_plane = I.in_plane = zplane;
    F.lout = g.nos[za];
    I.lin = g.nos[za];
    I.nplanes = (int)bk;
    float2 *z = g.ndim == 3 ? zgrid : rows;
    F.src = image;
    F.dst = z;
    I.src = z;
    I.dst = out;
    I.factor = (float)(1.0 / (double)g.gvol);  // of the two transforms
    int st = launch_col(F, kImageIn, s);
    if (st) return st;
    ColPass Y{};
    if (g.ndim == 3) {
        Y.fa = g.ax[1];
        Y.X = (int)N0;
        Y.nplanes = (int)P;
        Y.nmid = (int)n2;
        Y.in_ax = Y.out_ax = N0;
        Y.lin = (int)N1;
        Y.lout = (int)n1;
        Y.in_plane = n2 * N1 * N0;
        Y.in_mid = N1 * N0;
        Y.out_plane = n2 * n1 * N0;
        Y.out_mid = n1 * N0;
        Y.src = zgrid;
        Y.dst = rows;
        if ((st = launch_col(Y, kForward, s))) return st;
    }
    GramRows R{};
    R.fa = g.ax[0];
    R.N0 = (int)N0;
    R.rows = (int)(n1 * n2);
    R.K = g.K;
    R.lowrank = g.lowrank;
    R.batch = (int)batch;
    R.nseg = g.nseg;
    R.gvol = g.gvol;
    R.kern = g.kern;
    R.grid = rows;
    if ((st = launch_gram_rows(R, s))) return st;
    if (g.ndim == 3) {
        std::swap(Y.lin, Y.lout);
        std::swap(Y.in_plane, Y.out_plane);
        std::swap(Y.in_mid, Y.out_mid);
        Y.src = rows;
        Y.dst = zgrid;
        if ((st = launch_col(Y, kInverse, s))) return st;
    }
    return launch_col(I, kImageOut, s);
}

}  // namespace pfb
