// TMA form of two fused FFT passes, for the transform lengths with a compile-time stage
// plan (250 = 25 x 10, 240 = 16 x 15, 160 = 16 x 10, 256 = 16 x 16): the last pass of the
// adjoint (columns of the grid to the image) and the forward's x pass (rows to the
// channel-interleaved grid).  Persistent CTAs walk tiles of 16 vectors that the tensor
// memory accelerator loads into a two-slot ring while the previous tile transforms, stage by
// stage in shared memory.  The other passes run faster in the direct form (tma_pass).
#include <cuda.h>

#include "pfb_fft_passes.cuh"

namespace pfb {
namespace fft {
namespace {

constexpr int kCols = 16;                 // vectors per CTA
constexpr int kThreads = 256;
constexpr int kPairStreams = kThreads / (kCols / 2);  // butterflies: a thread takes 2 columns

// at most 256 (kTmaMax): a tile's rows are one box
constexpr int kTmaMax = 256;
constexpr bool tma_length(int n) { return n == 250 || n == 240 || n == 160 || n == 256; }
struct StagePlan {
    int radix[2];
};
constexpr StagePlan stage_plan(int n) {
    return n == 250 ? StagePlan{{25, 10}} : n == 240 ? StagePlan{{16, 15}} : n == 160 ? StagePlan{{16, 10}} : StagePlan{{16, 16}};
}

// Source of a stage: position pos of the column pair cp as (col 2cp, col 2cp + 1).
// Rows of PITCH float2, position-major (the layout every stage writes).
template <int PITCH>
struct PitchLoad {
    const float2 *src;
    __device__ __forceinline__ float4 operator()(int pos, int cp) const {
        return *reinterpret_cast<const float4 *>(src + pos * PITCH + 2 * cp);
    }
    // position pos of column c alone
    __device__ __forceinline__ float2 one(int pos, int c) const { return src[pos * PITCH + c]; }
};

// Source of the first stage of an x pass: 16 rows (one per vector) of `pitch`
// float2 as loaded from global memory (row-major); position pos holds element
// x = (pos + rot) mod n of its row, zero where x >= len (the pruned input)
struct RowMajorLoad {
    const float2 *src;
    int pitch, n, rot, len;
    __device__ __forceinline__ float2 one(int pos, int c) const {
        int x = pos + rot;
        if (x >= n) x -= n;
        if (x >= len) return make_float2(0.f, 0.f);
        return src[c * pitch + x];
    }
};

// Radices whose stages run with one column per thread (16 columns x 16 butterfly
// streams): a butterfly of two columns would hold 30 to 50 complex values
constexpr bool one_col_radix(int r) { return r >= 15; }
constexpr int kColStreams = kThreads / kCols;

// A Stockham stage with one column per thread: thread t takes column t mod 16 of
// butterflies t / 16, t / 16 + 16, ...  Same positions, twiddles and results as
// the two-column form.
template <int R, int NS, int M, int PITCH, class L>
__device__ __forceinline__ void fft_stage1_cl(const L &ld, float2 *__restrict__ dst, const float2 *__restrict__ tw) {
    constexpr int IT = (M + kColStreams - 1) / kColStreams;
    const int c = threadIdx.x & (kCols - 1), stream = threadIdx.x / kCols;
#pragma unroll
    for (int it = 0; it < IT; ++it) {
        const int i = stream + it * kColStreams;
        if (M % kColStreams != 0 && i >= M) break;
        const int j = NS == 1 ? 0 : i % NS;
        float2 a[R];
#pragma unroll
        for (int q = 0; q < R; ++q) a[q] = ld.one(i + q * M, c);
        if (NS > 1 && j != 0) {
#pragma unroll
            for (int q = 1; q < R; ++q) a[q] = cmul(a[q], __ldg(tw + (q - 1) * NS + j));
        }
        dft<R>(a);
        const int base = (i - j) * R + j;
#pragma unroll
        for (int k = 0; k < R; ++k) dst[(base + k * NS) * PITCH + c] = a[k];
    }
}

template <int R, int NS, int M, int PITCH, class L>
__device__ __forceinline__ void fft_stage_cl(const L &ld, float2 *__restrict__ dst, const float2 *__restrict__ tw,
                                             int stream, int cp) {
    constexpr int IT = (M + kPairStreams - 1) / kPairStreams;
#pragma unroll
    for (int it = 0; it < IT; ++it) {
        const int i = stream + it * kPairStreams;
        if (M % kPairStreams != 0 && i >= M) break;
        const int j = NS == 1 ? 0 : i % NS;
        float2 a[R], b[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const float4 v = ld(i + q * M, cp);
            a[q] = make_float2(v.x, v.y);
            b[q] = make_float2(v.z, v.w);
        }
        if (NS > 1 && j != 0) {
#pragma unroll
            for (int q = 1; q < R; ++q) {
                const float2 w = __ldg(tw + (q - 1) * NS + j);
                a[q] = cmul(a[q], w);
                b[q] = cmul(b[q], w);
            }
        }
        dft<R>(a);
        dft<R>(b);
        const int base = (i - j) * R + j;
#pragma unroll
        for (int k = 0; k < R; ++k)
            *reinterpret_cast<float4 *>(dst + (base + k * NS) * PITCH + 2 * cp) =
                make_float4(a[k].x, a[k].y, b[k].x, b[k].y);
    }
}

// Forward FFT of length N of the CTA's 16 columns: the first stage reads its input through
// `ld` and writes B, the second writes A (rows PITCH float2 apart).  Ends with the CTA
// synchronised; returns A.
template <int N, int PITCH, class L>
__device__ __forceinline__ float2 *fft_run_n(const L &ld, float2 *A, float2 *B, const float2 *tw) {
    constexpr StagePlan SP = stage_plan(N);
    constexpr int R0 = SP.radix[0], R1 = SP.radix[1];
    const int cp = threadIdx.x & (kCols / 2 - 1), stream = threadIdx.x / (kCols / 2);
    if constexpr (one_col_radix(R0)) fft_stage1_cl<R0, 1, N / R0, PITCH>(ld, B, tw);
    else fft_stage_cl<R0, 1, N / R0, PITCH>(ld, B, tw, stream, cp);
    __syncthreads();
    const float2 *tw1 = tw + R0 - 1;  // after the first stage's (ns = 1) twiddles
    if constexpr (one_col_radix(R1)) fft_stage1_cl<R1, R0, N / R1, PITCH>(PitchLoad<PITCH>{B}, A, tw1);
    else fft_stage_cl<R1, R0, N / R1, PITCH>(PitchLoad<PITCH>{B}, A, tw1, stream, cp);
    __syncthreads();
    return A;
}

// nullptr for any other length (the caller only launches with these)
template <int PITCH, class L>
__device__ __forceinline__ float2 *fft_run(const L &ld, float2 *A, float2 *B, const FftAxis &fa) {
    switch (fa.n) {
        case 250: return fft_run_n<250, PITCH>(ld, A, B, fa.tw);
        case 240: return fft_run_n<240, PITCH>(ld, A, B, fa.tw);
        case 160: return fft_run_n<160, PITCH>(ld, A, B, fa.tw);
        case 256: return fft_run_n<256, PITCH>(ld, A, B, fa.tw);
        default: return nullptr;
    }
}

// ------------------------------------------------------------------------------------
// Last pass of the adjoint: columns of the grid (z in 3D, y in 2D) -> image.  A persistent
// CTA walks column tiles (16 adjacent x positions x the whole axis, one (mid, plane)), each
// loaded by TMA into one slot of a two-slot ring while the previous tile transforms.  Rows
// are dense in shared memory (16 float2 = 128 bytes, the box layout).  The forward transform
// runs and its output is read reversed, IDFT(x)[k] = DFT(x)[(n - k) mod n], which needs no
// conjugation of the input or output.
// ------------------------------------------------------------------------------------
constexpr int kTmaPitch = kCols;        // float2 per shared row: one 128-byte TMA box row
constexpr int kWaitLimit = 1 << 20;     // mbarrier polls before a wait gives up

struct ColTma {
    FftAxis fa;
    int lout, hn;           // rows written; rotation of the fftshift (N / 2)
    int X, nxc, nmid;
    int ntiles;             // output blocks (16 x positions of one (mid, plane))
    int nseg;               // tiles per output block: the B0 segments summed, else 1
    int64_t out_mid, out_ax;
    float2 *dst;
    Chan ch;
    int C;
    int64_t nvol;
    const float *apod_ax, *apod_mid, *apod_x;
    const float2 *Cl;       // B0 segment factors on the image side (nseg x nvol), in the SEG form
    float factor;
    int accumulate;
    int *err;               // set to 1 when a wait gives up (the results are then invalid)
};

__device__ __forceinline__ unsigned smem_u32(const void *p) {
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
// bounded wait for the phase with the given parity to complete
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, unsigned parity) {
    const unsigned a = smem_u32(bar);
    for (int it = 0; it < kWaitLimit; ++it) {
        unsigned done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}
// 4D tiled TMA load into this CTA's shared memory, completing on `bar`
__device__ __forceinline__ void tma_load4(void *dst, const CUtensorMap *map, int c0, int c1, int c2, int c3,
                                          uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
        : "memory");
}
// 4D tiled TMA store from shared memory (bulk-group completion)
__device__ __forceinline__ void tma_store4(const CUtensorMap *map, int c0, int c1, int c2, int c3, const void *src) {
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3, %4}], [%5];" ::"l"(map),
                 "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(src))
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read0() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

struct TileInfo {
    int xc, mid, plane, l;  // l: segment of an adjoint last pass (0 otherwise)
};

// src_map: the pass's source as 4D (2X floats, rows, mid, source plane).
// Two ring slots (the next tile loads while this one transforms; 2 CTAs per SM): one slot
// and 3 CTAs per SM took 1.30 against 1.21 ms for the 200^3 z pass.
// SEG: B0 factors and segment sums; the plain instantiation keeps its simpler loops.  The
// segments are summed in registers (added to the image one by one, 192^2 x 768 with 8
// segments of 240 points took 1072 us against 897; the factor loads have to be ahead of the
// products, 4 rows at a time: row by row 1418 us).
template <bool SEG>
__global__ void __launch_bounds__(kThreads, 2)
    col_tma_kernel(const __grid_constant__ CUtensorMap src_map, const ColTma P) {
    extern __shared__ __align__(128) float2 tsm[];
    __shared__ __align__(8) uint64_t full[2];
    __shared__ TileInfo info[2];
    const int n = P.fa.n;
    // slot s of the ring at tsm + s * n rows, the transform's scratch buffer after them
    float2 *scr = tsm + 2 * n * kTmaPitch;
    const int col = (threadIdx.x % (kCols / 2)) * 2, stream = threadIdx.x / (kCols / 2);
    constexpr int NS = kThreads * 2 / kCols;  // row streams: a thread moves two adjacent columns
    const unsigned box_bytes = (unsigned)n * kTmaPitch * sizeof(float2);
    // thread 0: load segment l of output block t into slot s (tile coordinates go with
    // it through shared memory)
    auto issue = [&](int t, int l, int s) {
        const int r = t / P.nxc, xc = t - r * P.nxc;
        const int plane = r / P.nmid, mid = r - plane * P.nmid;
        // image plane (b, c) <- grid plane (grp, chn) of segment l
        const int b = plane / P.C, c = plane - b * P.C;
        const int Kc = P.ch.K ? P.ch.K : 1;
        const int sp = (P.ch.K ? 0 : c) * P.ch.nch + (P.ch.K ? (l * P.ch.B + b) * Kc + c : l * P.ch.B + b);
        info[s] = TileInfo{xc, mid, plane, l};
        mbar_expect_tx(&full[s], box_bytes);
        tma_load4(tsm + s * n * kTmaPitch, &src_map, xc * 2 * kCols, 0, mid, sp, &full[s]);
    };
    // the CTA's k-th tile: segment k mod nseg of its output block k / nseg (the
    // segments of one block are consecutive, so one CTA sums them)
    auto block_of = [&](int kk, int &l) {
        const int q = SEG ? kk / P.nseg : kk;
        l = kk - q * P.nseg;
        return (int)blockIdx.x + q * (int)gridDim.x;
    };
    if (threadIdx.x == 0) {
        mbar_init(&full[0], 1);
        mbar_init(&full[1], 1);
        fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) {
            int l;
            const int t = block_of(s, l);
            if (t < P.ntiles) issue(t, l, s);
        }
    }
    constexpr int kRows = SEG ? kTmaMax / NS : 1;  // rows of a column pair that a thread writes
    float4 sum[kRows];
#pragma unroll
    for (int u = 0; u < kRows; ++u) sum[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = 0;; ++k) {
        int lk;
        const int t = block_of(k, lk);
        if (t >= P.ntiles) break;
        const int s = k & 1;
        bool ok = mbar_wait(&full[s], (k >> 1) & 1);
        const TileInfo ti = info[s];
        float2 *A = tsm + s * n * kTmaPitch;
        const int x = ti.xc * kCols + col;
        const bool xin = x < P.X;
        const int xs = xin ? x : P.X - 2;
        float amid0 = P.factor, amid1 = P.factor;
        if (P.apod_mid) {
            amid0 *= P.apod_mid[ti.mid];
            amid1 *= P.apod_mid[ti.mid];
        }
        if (P.apod_x) {
            amid0 *= P.apod_x[xs];
            amid1 *= P.apod_x[xs + 1];
        }
        // every thread agrees on the wait's outcome
        ok = __syncthreads_and(ok);
        if (!ok) {
            if (threadIdx.x == 0) {
                atomicExch(P.err, 1);
                // the other slot's load, if one is in flight
                int l1;
                if (block_of(k + 1, l1) < P.ntiles) mbar_wait(&full[s ^ 1], ((k + 1) >> 1) & 1);
            }
            return;
        }
        const float2 *R = fft_run<kTmaPitch>(PitchLoad<kTmaPitch>{A}, A, scr, P.fa);
        int ln;
        const int tn = block_of(k + 2, ln);  // the next tile for this slot
        // output row o holds inverse-transform position pp = (o - hn) mod n, i.e. the
        // forward transform's position (n - pp) mod n
        const int64_t obase = (int64_t)ti.plane * P.nvol + (int64_t)ti.mid * P.out_mid;
        if (SEG) {
            // the segments of the block are summed in registers: kRows rows of two columns
            const float2 *clp = P.Cl + (int64_t)ti.l * P.nvol + (int64_t)ti.mid * P.out_mid + xs;
            // kU rows at a time: their factor loads are in flight before the first product
            constexpr int kU = 4;
#pragma unroll
            for (int u0 = 0; u0 < kRows; u0 += kU) {
                float4 cc[kU];
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    const int o = min(stream + (u0 + u) * NS, P.lout - 1);
                    cc[u] = __ldg(reinterpret_cast<const float4 *>(clp + (int64_t)o * P.out_ax));
                }
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    const int o = min(stream + (u0 + u) * NS, P.lout - 1);
                    int pp = o - P.hn;
                    if (pp < 0) pp += n;
                    const int q = pp == 0 ? 0 : n - pp;
                    const float4 w = *reinterpret_cast<const float4 *>(R + q * kTmaPitch + col);
                    // times conj(C_l) of the tile's segment
                    const float2 v0 = cmulc(make_float2(w.x, w.y), make_float2(cc[u].x, cc[u].y));
                    const float2 v1 = cmulc(make_float2(w.z, w.w), make_float2(cc[u].z, cc[u].w));
                    float4 &t = sum[u0 + u];
                    t.x += v0.x;
                    t.y += v0.y;
                    t.z += v1.x;
                    t.w += v1.y;
                }
            }
            if (ti.l + 1 == P.nseg) {
#pragma unroll
                for (int u = 0; u < kRows; ++u) {
                    const int o = stream + u * NS;
                    float4 w = sum[u];
                    sum[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (o >= P.lout || !xin) continue;
                    const float a = P.apod_ax ? P.apod_ax[o] : 1.f;
                    const float a0 = a * amid0, a1 = a * amid1;
                    float4 *d = reinterpret_cast<float4 *>(P.dst + obase + (int64_t)o * P.out_ax + x);
                    w.x *= a0;
                    w.y *= a0;
                    w.z *= a1;
                    w.w *= a1;
                    if (P.accumulate) {
                        const float4 old = *d;
                        w.x += old.x;
                        w.y += old.y;
                        w.z += old.z;
                        w.w += old.w;
                    }
                    *d = w;
                }
            }
        } else {
            for (int o = stream; o < P.lout; o += NS) {
                int pp = o - P.hn;
                if (pp < 0) pp += n;
                const int q = pp == 0 ? 0 : n - pp;
                float4 v = *reinterpret_cast<const float4 *>(R + q * kTmaPitch + col);
                if (!xin) continue;
                float4 *d = reinterpret_cast<float4 *>(P.dst + obase + (int64_t)o * P.out_ax + x);
                const float a = P.apod_ax ? P.apod_ax[o] : 1.f;
                const float a0 = a * amid0, a1 = a * amid1;
                v.x *= a0;
                v.y *= a0;
                v.z *= a1;
                v.w *= a1;
                if (P.accumulate) {
                    const float4 old = *d;
                    v.x += old.x;
                    v.y += old.y;
                    v.z += old.z;
                    v.w += old.w;
                }
                *d = v;
            }
        }
        // the slot and the scratch buffer are read; the generic accesses are ordered
        // before the slot's next TMA load
        fence_async_smem();
        __syncthreads();
        // refill this slot with the tile after next
        if (threadIdx.x == 0 && tn < P.ntiles) issue(tn, ln, s);
    }
}

// ------------------------------------------------------------------------------------
// Forward x pass on TMA.  A tile is 16 consecutive vectors (rows along x); each row arrives
// by tensor-map boxes, `pitch` float2 apart in shared memory, into one slot of a two-slot
// ring while the previous tile transforms.  The first radix stage reads that row-major
// layout (RowMajorLoad: the fftshift rotation and the zero padding fold into its index) and
// writes the position-major layout of the later stages: rows of T (N0 long,
// [plane][kz][ky][x]) -> the interleaved grid, the 16 vectors being 16 consecutive channels
// of one (group, kz, ky), stored by TMA as boxes of 16 channels x kx (rows 16 float2 wide).
// ------------------------------------------------------------------------------------
struct RowTma {
    FftAxis fa;
    int len, rot;       // input row length; first-stage rotation N0 / 2
    int ntiles;
    int nch, nos1, nos2;
    int pitch;          // x extent of the load box = float2 between the loaded rows (>= len;
                        // the columns past len are zero-filled)
    int slot;           // float2 per ring slot
    int *err;
};

__device__ __forceinline__ void tma_load3(void *dst, const CUtensorMap *map, int c0, int c1, int c2, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
        : "memory");
}

__global__ void __launch_bounds__(kThreads, 2)
    row_tma_kernel(const __grid_constant__ CUtensorMap src_map, const __grid_constant__ CUtensorMap dst_map,
                   const RowTma P) {
    constexpr int PITCH = kTmaPitch;
    extern __shared__ __align__(128) float2 tsm[];
    __shared__ __align__(8) uint64_t full[2];
    const int n = P.fa.n;
    float2 *scr = tsm + 2 * P.slot;
    // thread 0: load tile t into slot s as one box of 16 rows of P.pitch (rows past the
    // last vector and columns past the row length are zero-filled).  A tensor copy's
    // shared-memory destination must be 128-byte aligned: the slots are; a slot that
    // is not (never by construction) sets the error flag and is not loaded
    auto issue = [&](int t, int s) {
        float2 *dst = tsm + s * P.slot;
        const int u0 = t * kCols;
        if (smem_u32(dst) & 127u) {
            atomicExch(P.err, 1);
            mbar_expect_tx(&full[s], 0);
            return;
        }
        mbar_expect_tx(&full[s], (unsigned)(kCols * P.pitch * sizeof(float2)));
        // 16 consecutive channels of one (group, kz, ky): planes grp nch + chn0 ..
        const int chn0 = u0 % P.nch;
        int r = u0 / P.nch;
        const int ky = r % P.nos1;
        r /= P.nos1;
        const int kz = r % P.nos2, grp = r / P.nos2;
        tma_load3(dst, &src_map, 0, kz * P.nos1 + ky, grp * P.nch + chn0, &full[s]);
    };
    if (threadIdx.x == 0) {
        mbar_init(&full[0], 1);
        mbar_init(&full[1], 1);
        fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) {
            const int t = blockIdx.x + s * gridDim.x;
            if (t < P.ntiles) issue(t, s);
        }
    }
    int k = 0;
    for (int t = blockIdx.x; t < P.ntiles; t += gridDim.x, ++k) {
        const int s = k & 1;
        bool ok = mbar_wait(&full[s], (k >> 1) & 1);
        float2 *S = tsm + s * P.slot;
        ok = __syncthreads_and(ok);
        if (!ok) {
            if (threadIdx.x == 0) {
                atomicExch(P.err, 1);
                if (t + (int)gridDim.x < P.ntiles) mbar_wait(&full[s ^ 1], ((k + 1) >> 1) & 1);
            }
            return;
        }
        const RowMajorLoad ld{S, P.pitch, n, P.rot, P.len};
        const float2 *R = fft_run<PITCH>(ld, S, scr, P.fa);
        const int u0 = t * kCols;
        const int tn = t + 2 * gridDim.x;
        // rows kx of the result are 16 channels of point (kz, ky, kx): TMA store
        fence_async_smem();
        __syncthreads();
        if (threadIdx.x == 0) {
            const int chn0 = u0 % P.nch;
            int r = u0 / P.nch;
            const int ky = r % P.nos1;
            r /= P.nos1;
            const int kz = r % P.nos2, grp = r / P.nos2;
            tma_store4(&dst_map, chn0, 0, kz * P.nos1 + ky, grp, R);
            bulk_commit();
            // a two-stage transform leaves its result in the slot: refill it once the store
            // has read it
            bulk_wait_read0();
            if (tn < P.ntiles) issue(tn, s);
        }
    }
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (the driver
// library itself is not linked)
using EncodeTiledFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                   const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled() {
    static const EncodeTiledFn fn = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            f = nullptr;
        return reinterpret_cast<EncodeTiledFn>(f);
    }();
    return fn;
}

// 4D map over complex64 data seen as float32 pairs: (2 X floats, rows, mid,
// planes) with the given element strides, boxes of 16 complex x br rows.  Rows
// past `rows` read as zeros.  Strides of unit extents are unused: any legal value.
bool encode_col_map(CUtensorMap *m, const void *base, int X, int rows, int nmid, int64_t nplanes, int64_t s_row,
                    int64_t s_mid, int64_t s_plane, int br) {
    const EncodeTiledFn fn = encode_tiled();
    if (!fn) return false;
    if (nmid == 1) s_mid = s_row;
    if (nplanes == 1) s_plane = s_row;
    const cuuint64_t dim[4] = {(cuuint64_t)2 * X, (cuuint64_t)rows, (cuuint64_t)nmid, (cuuint64_t)nplanes};
    const cuuint64_t str[3] = {(cuuint64_t)s_row * 8, (cuuint64_t)s_mid * 8, (cuuint64_t)s_plane * 8};
    for (cuuint64_t v : str)
        if (v == 0 || v % 16 != 0 || v >= (1ull << 40)) return false;
    const cuuint32_t box[4] = {2 * kCols, (cuuint32_t)br, 1, 1};
    const cuuint32_t es[4] = {1, 1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<void *>(base), dim, str, box, es,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Which passes run here; the others took, TMA against direct, in us (200^3 at osf 1.25 with
// 32 coils; 192^2 at 1.25 with 6 segments of 12 coils; 128^3 at 1.25 with 32; 128^2 at 2
// with 64):
//              250          240          160        256
//   x fwd      1477 / 2052  922 / 1110   407 / 432  674 / 763    here
//   image out  1178 / 1262   897 / 1536  303 / 270  5.8 / 6.4    here but 160
//   image in   1114 / 1067  1278 / 858   330 / 280               direct
//   y fwd      1117 / 1111               307 / 286               direct
//   y inv      1231 / 1079               326 / 260               direct
//   x inv      1632 / 1588  1036 / 794   426 / 343               direct
bool tma_pass(int n, int pass) {
    return tma_length(n) && (pass == kRowForward || (pass == kImageOut && n != 160));
}

// Tiled tensor map over 8-byte elements (complex64 as one element): rank dims
// (innermost first), rank - 1 byte strides, a box per dimension.  Rows past an
// extent read as zeros.
bool encode_map8(CUtensorMap *m, const void *base, int rank, const cuuint64_t *dim, const cuuint64_t *stride,
                 const cuuint32_t *box) {
    const EncodeTiledFn fn = encode_tiled();
    if (!fn || rank < 1 || rank > 5) return false;
    for (int i = 0; i < rank - 1; ++i)
        if (stride[i] == 0 || stride[i] % 16 != 0 || stride[i] >= (1ull << 40)) return false;
    for (int i = 0; i < rank; ++i)
        if (dim[i] == 0 || box[i] == 0 || box[i] > 256) return false;
    if ((box[0] * 8) % 16 != 0) return false;
    const cuuint32_t es[5] = {1, 1, 1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_INT64, (cuuint32_t)rank, const_cast<void *>(base), dim, stride, box, es,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

// The adjoint's last pass on TMA when its layout allows it (every stride and base 16-byte
// aligned, even X); returns 1 if launched, 0 to take the direct form, or an error.  The
// segments of an output block are consecutive tiles of one CTA.
int launch_col_tma(const ColPass &P, int pass, cudaStream_t s) {
    const int n = P.fa.n;
    if (!P.err || P.nsm <= 0 || P.X % 2 != 0 || !tma_pass(n, pass)) return 0;
    const int64_t ntiles = (int64_t)P.nplanes * P.nmid * ((P.X + kCols - 1) / kCols);
    auto a16 = [](const void *q) { return ((uintptr_t)q & 15u) == 0; };
    if (!a16(P.src) || !a16(P.dst)) return 0;
    if (P.Cl && !a16(P.Cl)) return 0;
    if (P.ch.L < 1 || (P.ch.L > 1 && !P.Cl)) return 0;
    for (int64_t v : {P.in_ax, P.in_mid, P.in_plane, P.out_ax, P.out_mid, P.nvol})
        if (v % 2 != 0) return 0;
    ColTma T{};
    T.fa = P.fa;
    T.lout = P.lout;
    T.hn = P.nax / 2;
    T.X = P.X;
    T.nxc = (P.X + kCols - 1) / kCols;
    T.nmid = P.nmid;
    if (ntiles >= (1LL << 31) - 2LL * P.nsm * 4) return 0;
    T.ntiles = (int)ntiles;
    T.nseg = P.ch.L;
    if (P.lin != n) return 0;
    T.out_mid = P.out_mid;
    T.out_ax = P.out_ax;
    T.dst = P.dst;
    T.ch = P.ch;
    T.C = P.C;
    T.nvol = P.nvol;
    T.apod_ax = P.apod_ax;
    T.apod_mid = P.apod_mid;
    T.apod_x = P.apod_x;
    T.Cl = P.Cl;
    T.factor = P.factor;
    T.accumulate = P.accumulate;
    T.err = P.err;
    CUtensorMap smap;
    if (!encode_col_map(&smap, P.src, P.X, n, P.nmid, (int64_t)P.ch.ngrp * P.ch.nch, P.in_ax, P.in_mid, P.in_plane,
                        n))
        return 0;
    const size_t smem = (size_t)3 * n * kTmaPitch * sizeof(float2);
    auto kern = P.Cl ? col_tma_kernel<true> : col_tma_kernel<false>;
    PFB_RAISE_SMEM(kern, (int)smem);
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, smem) != cudaSuccess || per_sm < 1)
        return 0;
    const int64_t grid = std::min<int64_t>(ntiles, (int64_t)P.nsm * per_sm);
    kern<<<(unsigned)grid, kThreads, smem, s>>>(smap, T);
    PFB_CHECK_LAUNCH();
    return 1;
}

// The forward x pass on TMA when the layout allows it (a length of tma_pass, even row
// lengths, 16-byte aligned bases, 32-bit vector indices, a multiple of 16 channels); returns
// 1 if launched, 0 to take the direct form, or an error.
int launch_row_tma(const RowPass &P, bool inv, cudaStream_t s) {
    const int n = P.fa.n;
    if (!P.err || P.nsm <= 0 || !tma_pass(n, inv ? kRowInverse : kRowForward) || P.N0 % 2 != 0) return 0;
    if (P.nvec <= 0 || P.nvec >= (1LL << 31) - (int64_t)kCols * 4 * P.nsm) return 0;
    if (P.nch % kCols != 0) return 0;
    auto a16 = [](const void *q) { return ((uintptr_t)q & 15u) == 0; };
    if (!a16(P.src) || !a16(P.dst)) return 0;
    RowTma T{};
    T.fa = P.fa;
    T.len = P.N0;
    T.rot = P.N0 / 2;
    T.ntiles = (int)((P.nvec + kCols - 1) / kCols);
    T.nch = P.nch;
    T.nos1 = P.nos1;
    T.nos2 = P.nos2;
    // one box per tile, x extent = row pitch >= the row length with pitch = 2 (mod 8):
    // the first stage's column reads (8 column pairs x 4 positions per warp) then touch
    // each bank at most twice; a box is at most 256 wide
    T.pitch = T.len;
    while (T.pitch % 8 != 2) ++T.pitch;
    if (T.pitch > 256) return 0;
    T.slot = std::max(kCols * T.pitch, n * kTmaPitch);
    T.slot = (T.slot + 15) / 16 * 16;  // 128-byte aligned slots
    T.err = P.err;
    CUtensorMap smap, dmap;
    // rows of T: x, row (kz, ky) of a plane, plane (group, channel); 16 planes per tile
    const int64_t planes = P.nvec / ((int64_t)P.nos1 * P.nos2);
    const cuuint64_t dim[3] = {(cuuint64_t)P.N0, (cuuint64_t)P.nos2 * P.nos1, (cuuint64_t)planes};
    const cuuint64_t str[2] = {(cuuint64_t)P.N0 * 8, (cuuint64_t)P.N0 * P.nos2 * P.nos1 * 8};
    const cuuint32_t box[3] = {(cuuint32_t)T.pitch, 1, (cuuint32_t)kCols};
    if (!encode_map8(&smap, P.src, 3, dim, str, box)) return 0;
    const int64_t ngrp = planes / P.nch;
    const cuuint64_t odim[4] = {(cuuint64_t)P.nch, (cuuint64_t)n, (cuuint64_t)P.nos2 * P.nos1, (cuuint64_t)ngrp};
    const cuuint64_t ostr[3] = {(cuuint64_t)P.nch * 8, (cuuint64_t)n * P.nch * 8, (cuuint64_t)P.gvol * P.nch * 8};
    const cuuint32_t obox[4] = {(cuuint32_t)kCols, (cuuint32_t)n, 1, 1};
    if (!encode_map8(&dmap, P.dst, 4, odim, ostr, obox)) return 0;
    const size_t smem = (size_t)3 * T.slot * sizeof(float2);
    auto k = row_tma_kernel;
    PFB_RAISE_SMEM(k, (int)smem);
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kThreads, smem) != cudaSuccess || per_sm < 1)
        return 0;
    const int grid = (int)std::min<int64_t>(T.ntiles, (int64_t)P.nsm * per_sm);
    k<<<grid, kThreads, smem, s>>>(smap, dmap, T);
    PFB_CHECK_LAUNCH();
    return 1;
}

}  // namespace fft
}  // namespace pfb
