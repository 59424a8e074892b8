// Plain FP64 GEMM on the sm_100a FP64 tensor path (DMMA, mma.sync m16n8k4 f64),
// fed by TMA through a multi-stage mbarrier pipeline, as one persistent
// grouped launch over every tile of every problem.
//
// Replaces the reference's per-Cannon-step cublasDgemm + stream sync
// (src/cannon.c:410-418, :651-676; src/cuda_proxy.cu:211-230).  All virtual
// ranks' cuboid GEMMs of one ca3dmm exec run in this single launch -- or, for a
// product of few tiles, as k segments of its tiles shared out evenly (below).
//
// Layout (per stage, 32 KiB for 128-column tiles or 24 KiB for 64-column
// ones, 1024-byte aligned):
//   A tile: 128 (m) x 16 (k) doubles as 8 TMA boxes of 16 m x 16 k, each box
//           16 rows (k) of 128 B (m), SWIZZLE_128B -- or, for a K-major A
//           (a transposed operand read in place), 1 box of 128 rows (m) of
//           128 B (k), like B.
//   B tile: TBN (n) x 16 (k) doubles as 1 TMA box, TBN rows (n) of 128 B (k),
//           SWIZZLE_128B (TBN = 128 or 64 output columns per tile).
// Fragment ownership is permuted so every fragment load is one conflict-free
// 128-bit LDS:
//   * MMA row r of an m16 tile  -> tile row 2r (r < 8) or 2(r-8)+1, so a0/a1 of
//     m16n8k4 are the two doubles of one 16-byte chunk;
//   * MMA column c of n8 tile j -> warp column 4c + j;
//   * MMA k index t of k-step (q, b) -> tile k row 8q + 2t + b, so one 16-byte
//     chunk of a B row holds the b0 fragments of two consecutive k-steps.
// With the 128B swizzle (16-byte chunk index XOR row % 8) these choices put
// every quarter-warp of a 128-bit load on 8 distinct chunks.
// K-major A: a 16-byte chunk of a tile row holds that row's a0 (or a1) of two
// consecutive k-steps, as for B.  MMA rows g and g + 8 of m16 tile i are tile
// rows 16i + 2 sigma(g) and 16i + 2 sigma(g) + 1, sigma swapping the two low
// bits of g, so the two rows of a quarter-warp differ by 4 (mod 8) and hit
// disjoint chunk sets, and the C pairs (m, m+1) stay adjacent.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <atomic>
#include "k_common.cuh"
#include "ca3dmm_kernels.h"

namespace {

constexpr int BM = 128, BK = 16;
constexpr int A_BYTES = BM * BK * 8;                 // 16 KiB
constexpr int CONSUMER_WARPS = 8;
constexpr int THREADS = CONSUMER_WARPS * 32;         // thread 0 also issues the TMA loads
constexpr int GROUP_M = 8;

// The output tile is BM x TBN, TBN = 128 or 64 columns.  Each warp computes
// 16 MI rows x 32 columns (MI m16 tiles x 4 n8 tiles): the 8 warps stand
// WM x WN = 2 x 4 over a 128-column tile and 4 x 2 over a 64-column one, so
// the fragment layout of a warp is the same for both widths.
template <int TBN>
struct DTile {
    static_assert(TBN == 128 || TBN == 64, "tile width");
    static constexpr int WN = TBN / 32, WM = CONSUMER_WARPS / WN, MI = BM / (16 * WM);
    static constexpr int STAGE_BYTES = A_BYTES + TBN * BK * 8;   // 32 or 24 KiB
    static constexpr int STAGES = TBN == 128 ? 5 : 6;
    static constexpr size_t SMEM_BYTES = (size_t) STAGES * STAGE_BYTES + 2 * STAGES * 8 + 1024;
};

struct alignas(16) DProb {
    double *C;
    long long ldc;
    int m, n, k;
    int tiles_m, tiles_n, tile_begin;
    double alpha, beta;
    int vec_ok, raster;
};

// The problem holding tile `tile`.  sb: a shared-memory copy of the problems'
// first tiles (nullptr when there are more than PROB_CACHE problems), so that a
// batch of small GEMMs does not pay a chain of dependent global loads per tile.
constexpr int PROB_CACHE = 1024;
__device__ __forceinline__ int find_problem(const int *sb, const DProb *probs, int nprob, int tile)
{
    int lo = 0, hi = nprob - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if ((sb ? sb[mid] : probs[mid].tile_begin) <= tile) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ void tile_coords(const DProb &p, int tile, int &tm, int &tn)
{
    int t = tile - p.tile_begin;
    int group_size = p.raster * p.tiles_n;
    int group = t / group_size;
    int first_m = group * p.raster;
    int gm = min(p.tiles_m - first_m, p.raster);
    int r = t % group_size;
    tm = first_m + r % gm;
    tn = r / gm;
}

__device__ __forceinline__ void dmma(double (&d)[4], double a0, double a1, double b0)
{
    asm volatile(
        "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
        "{%0,%1,%2,%3};\n"
        : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
        : "d"(a0), "d"(a1), "d"(b0));
}

// Rows m, m + 1 of one column, alpha v + beta C.
__device__ __forceinline__ void store_pair(double *c, bool two, bool vec, double alpha, double beta,
                                           double v0, double v1)
{
    if (vec && two) {
        double2 o;
        if (beta != 0.0) {
            double2 old = *reinterpret_cast<const double2 *>(c);
            o.x = alpha * v0 + beta * old.x;
            o.y = alpha * v1 + beta * old.y;
        } else {
            o.x = alpha * v0;
            o.y = alpha * v1;
        }
        *reinterpret_cast<double2 *>(c) = o;
    } else {
        c[0] = beta != 0.0 ? alpha * v0 + beta * c[0] : alpha * v0;
        if (two) c[1] = beta != 0.0 ? alpha * v1 + beta * c[1] : alpha * v1;
    }
}

// This thread's part of a finished tile: its first row mb, first column nb.
// The problem's fields are read once into registers: read through the pointer
// they were loaded again after each of the 32 stores (which may alias them),
// 6-7 us per tile instead of 2-4.
template <int MI>
__device__ __forceinline__ void store_tile(const DProb &prob, int mb, int nb,
                                           const double (&acc)[MI][4][4])
{
    const int m = prob.m, n = prob.n;
    const bool vec = prob.vec_ok;
    const double alpha = prob.alpha, beta = prob.beta;
    const long long ldc = prob.ldc;
    double *c0 = prob.C + (long long) mb + (long long) nb * ldc;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (nb + j >= n) break;
        double *c = c0 + j * ldc;
#pragma unroll
        for (int i = 0; i < MI; ++i) {
            const int r = mb + 16 * i;
            if (r >= m) break;
            store_pair(c + 16 * i, r + 1 < m, vec, alpha, beta,
                       j < 4 ? acc[i][j & 3][0] : acc[i][j & 3][1],
                       j < 4 ? acc[i][j & 3][2] : acc[i][j & 3][3]);
        }
    }
}

// Iterator over this CTA's (tile, k-tile) load sequence, used by the
// producer thread.  Tiles with k == 0 carry no loads and are skipped.
template <int TBN>
struct LoadCursor {
    int tile, kt, ktiles, pi, m0, n0;   // tile: virtual index into the launch's ranges
    bool valid;
    __device__ void seek(const int *sb, const DProb *probs, int nprob,
                         const ca3dmm_tile_ranges_t &rg, int total_tiles, int stride)
    {
        while (tile < total_tiles) {
            const int t = range_tile(rg, tile);
            pi = find_problem(sb, probs, nprob, t);
            const DProb &p = probs[pi];
            ktiles = (p.k + BK - 1) / BK;
            if (ktiles > 0) {
                int tm, tn;
                tile_coords(p, t, tm, tn);
                m0 = tm * BM;
                n0 = tn * TBN;
                valid = true;
                return;
            }
            tile += stride;
        }
        valid = false;
    }
    __device__ void advance(const int *sb, const DProb *probs, int nprob,
                            const ca3dmm_tile_ranges_t &rg,
                            int total_tiles, int stride)
    {
        if (++kt < ktiles) return;
        kt = 0;
        tile += stride;
        seek(sb, probs, nprob, rg, total_tiles, stride);
    }
};

// sigma: swap the two low bits of g (0..7)
__device__ __forceinline__ int sigma_row(int g) { return (g & 4) | ((g & 1) << 1) | ((g >> 1) & 1); }

// The k loop of one output tile: wait for each stage, run the 16-k block's
// DMMAs, release the stage and (thread 0) refill it.  AK: A tile K-major.
template <bool AK, int TBN, class Issue>
__device__ __forceinline__ bool k_loop(const uint8_t *smem, uint64_t *full, uint64_t *empty,
                                       int ktiles, uint32_t &it,
                                       double (&acc)[DTile<TBN>::MI][4][4],
                                       volatile int *abort_flag, int *status,
                                       unsigned long long limit_ns, bool producer,
                                       Issue &issue_one, int wm, int wn, int g, int t, int lane)
{
    using T = DTile<TBN>;
    constexpr int MI = T::MI;
    for (int kt = 0; kt < ktiles; ++kt, ++it) {
        const uint32_t stage = it % T::STAGES, phase = (it / T::STAGES) & 1u;
        if (!mbar_wait_warp(&full[stage], phase, abort_flag, status, CA3DMM_DEV_TIMEOUT_CONSUME,
                            limit_ns))
            return false;
        const uint8_t *sA = smem + stage * T::STAGE_BYTES;
        const uint8_t *sB = sA + A_BYTES;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            double2 bf[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int nl = wn * 32 + 4 * g + j;
                bf[j] = *reinterpret_cast<const double2 *>(
                    sB + nl * 128 + (((4 * q + t) ^ (nl & 7)) << 4));
            }
            if (AK) {
#pragma unroll
                for (int ip = 0; ip < MI / 2; ++ip) {
                    double2 alo[2], ahi[2];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        // K-major A: tile row of MMA row g of m16 tile i
                        const int ra = wm * 16 * MI + 2 * sigma_row(g) + 16 * (2 * ip + h);
                        alo[h] = *reinterpret_cast<const double2 *>(
                            sA + ra * 128 + (((4 * q + t) ^ (ra & 7)) << 4));
                        ahi[h] = *reinterpret_cast<const double2 *>(
                            sA + (ra + 1) * 128 + (((4 * q + t) ^ ((ra + 1) & 7)) << 4));
                    }
#pragma unroll
                    for (int b = 0; b < 2; ++b)
#pragma unroll
                        for (int h = 0; h < 2; ++h)
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                dmma(acc[2 * ip + h][j], b ? alo[h].y : alo[h].x,
                                     b ? ahi[h].y : ahi[h].x, b ? bf[j].y : bf[j].x);
                    
                }
            } else {
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const int kr = 8 * q + 2 * t + b;
                    double2 af[MI];
#pragma unroll
                    for (int i = 0; i < MI; ++i)
                        af[i] = *reinterpret_cast<const double2 *>(
                            sA + (wm * MI + i) * 2048 + kr * 128 + ((g ^ (kr & 7)) << 4));
#pragma unroll
                    for (int i = 0; i < MI; ++i)
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            dmma(acc[i][j], af[i].x, af[i].y, b ? bf[j].y : bf[j].x);
                }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[stage]);
        // a refill that gives up has raised the abort flag: the wait for the missing
        // load ends the loop, for the whole warp
        if (producer) issue_one();
    }
    __syncwarp();
    return true;
}

// All 8 warps compute; thread 0 also drives the TMA pipeline.  Load L lands
// in stage L % STAGES; before issuing it the producer waits for the release
// of load L - STAGES.  Loads are issued STAGES-1 ahead of consumption, and the
// refill after consuming load `it` waits on the release of load it - 1, which
// every warp has usually finished, so the producer thread rarely stalls.
template <bool AK, int TBN>
__global__ void __launch_bounds__(THREADS, 1)
dgemm_dmma_grouped(const CUtensorMap *__restrict__ tmaps, const DProb *__restrict__ probs,
                   int nprob, const ca3dmm_tile_ranges_t rg, int total_tiles, int *status,
                   unsigned long long limit_ns)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    using T = DTile<TBN>;
    constexpr int STAGES = T::STAGES, STAGE_BYTES = T::STAGE_BYTES, MI = T::MI;
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + STAGES * STAGE_BYTES);
    uint64_t *empty = full + STAGES;
    __shared__ volatile int abort_flag;
    __shared__ int s_pbeg[PROB_CACHE];
    // the search table: rematerialised at each use (a kernel parameter and a
    // shared address), not held in a register across the main loop
#define CA3DMM_PB (nprob <= PROB_CACHE ? s_pbeg : nullptr)
    if (nprob <= PROB_CACHE)
        for (int i = threadIdx.x; i < nprob; i += blockDim.x) s_pbeg[i] = probs[i].tile_begin;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool producer = threadIdx.x == 0;
    if (producer) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], CONSUMER_WARPS);
        }
        abort_flag = 0;
        fence_barrier_init();
    }
    __syncthreads();

    LoadCursor<TBN> lc = {};
    uint32_t issued = 0;
    int last_p = -1;
    // Issue load number `issued` at the cursor (producer thread only).
    auto issue_one = [&]() -> bool {
        if (!lc.valid) return true;
        const uint32_t s = issued % STAGES, ph = (issued / STAGES) & 1u;
        if (!mbar_wait_bounded(&empty[s], ph ^ 1u, &abort_flag, status,
                               CA3DMM_DEV_TIMEOUT_PRODUCE, limit_ns))
            return false;
        const CUtensorMap *ta = tmaps + 2 * lc.pi, *tb = ta + 1;
        if (lc.pi != last_p) {
            tmap_acquire(ta);
            tmap_acquire(tb);
            last_p = lc.pi;
        }
        uint8_t *sA = smem + s * STAGE_BYTES;
        uint8_t *sB = sA + A_BYTES;
        mbar_arrive_expect_tx(&full[s], STAGE_BYTES);
        if (AK) {
            tma_load_2d(sA, ta, lc.kt * BK, lc.m0, &full[s]);
        } else {
#pragma unroll
            for (int j = 0; j < BM / 16; ++j)
                tma_load_2d(sA + j * 2048, ta, lc.m0 + 16 * j, lc.kt * BK, &full[s]);
        }
        tma_load_2d(sB, tb, lc.kt * BK, lc.n0, &full[s]);
        ++issued;
        lc.advance(CA3DMM_PB, probs, nprob, rg, total_tiles, gridDim.x);
        return true;
    };
    if (producer) {
        lc.tile = blockIdx.x;
        lc.kt = 0;
        lc.seek(CA3DMM_PB, probs, nprob, rg, total_tiles, gridDim.x);
        for (int s = 0; s < STAGES - 1; ++s)
            if (!issue_one()) break;
    }

    const int g = lane >> 2, t = lane & 3;
    const int wm = warp / T::WN, wn = warp % T::WN;
    uint32_t it = 0;   // loads consumed so far
    double acc[MI][4][4];
    bool ok = true;

    for (int v = blockIdx.x; v < total_tiles && ok; v += gridDim.x) {
        const int tile = range_tile(rg, v);
        int pi = find_problem(CA3DMM_PB, probs, nprob, tile);
        const DProb &p = probs[pi];
        int tm, tn;
        tile_coords(p, tile, tm, tn);
        const int ktiles = (p.k + BK - 1) / BK;
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0;

        ok = k_loop<AK, TBN>(smem, full, empty, ktiles, it, acc, &abort_flag, status, limit_ns,
                        producer, issue_one, wm, wn, g, t, lane);
        if (!ok) break;

        const int mb = tm * BM + wm * 16 * MI + 2 * (AK ? sigma_row(g) : g);
        const int nb = tn * TBN + wn * 32 + 8 * t;
        store_tile<MI>(p, mb, nb, acc);
    }

    if (producer) {
        // Wait (bounded, ignoring the abort flag) for every copy still in
        // flight so no TMA write lands in shared memory after exit.
        const uint32_t first = issued > STAGES ? issued - STAGES : 0;
        for (uint32_t L = first; L < issued; ++L) {
            const uint32_t s = L % STAGES, ph = (L / STAGES) & 1u;
            uint64_t t0 = global_timer_ns();
            while (!mbar_try_wait(&full[s], ph)) {
                if (global_timer_ns() - t0 > limit_ns) {
                    atomicCAS(status, 0, CA3DMM_DEV_TIMEOUT_PRODUCE);
                    break;
                }
            }
        }
    }
}
#undef CA3DMM_PB

// ------------------------------------------------------------------ k segments
// One problem whose tiles do not fill the chip evenly: the work list holds k
// segments of tiles instead of whole tiles (ca3dmm_dgemm_segments below), and a
// CTA runs the segments of its list in turn.  A tile cut into several segments
// is finished by whichever CTA completes its last one: every CTA writes its
// partial tile to the workspace and counts up the tile's counter, and the one
// that counts last adds the partials in segment order and stores C.  No CTA
// ever waits for another, and the order of the sum is fixed.
//
// Inside a segment the accumulators restart after at most CHUNK k tiles: the partial
// sums move to a running total in TMEM, which this kernel's MMAs leave free
// (the same thread writes and reads its words, 128 per thread at 128 columns).
// Rounding errors grow with the length of a chain of additions, so chunks of
// 256 k keep the result at least as accurate as the k sub-slabs of up to
// several thousand k, summed by a kernel of their own, that these shapes ran as
// before; the last chain but one of a longer segment has 128 k, which makes the sum of
// the squared lengths smaller whatever the rest is.
// All warps restart at the same block: the additions use the pipe of the
// MMAs, 1.3 us per chunk of 35 us (0.2 of it the moves to and from TMEM).  With the
// warps of rows 64 .. 127 half a chunk later they lost 1.8 us, with one m16 tile of
// a warp at a time, spread over the chunk, 5: an addition waits for the MMAs of the
// other warp (4736 x 1024 x 8192: 2364, 2427, 2674 us; without restarts 2277).
__device__ __forceinline__ void tmem_ld32_wait(uint32_t taddr, uint32_t (&v)[32])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
        "%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
          "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
          "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]),
          "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]),
          "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
        "%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]),
          "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]),
          "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]),
          "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]),
          "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}

// acc of m16 tile i (4 x 4 doubles = 32 words per thread) += its TMEM total
__device__ __forceinline__ void total_add(uint32_t taddr, double (&acc)[4][4])
{
    uint32_t v[32];
    tmem_ld32_wait(taddr, v);
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e)
            acc[j][e] = __hiloint2double((int) v[8 * j + 2 * e + 1], (int) v[8 * j + 2 * e]) + acc[j][e];
}

__device__ __forceinline__ void total_store(uint32_t taddr, const double (&acc)[4][4])
{
    uint32_t v[32];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            v[8 * j + 2 * e] = (uint32_t) __double2loint(acc[j][e]);
            v[8 * j + 2 * e + 1] = (uint32_t) __double2hiint(acc[j][e]);
        }
    tmem_st32(taddr, v);
}

// Order of a launch: CTA b runs segments begin[b] .. begin[b + 1] - 1 (the
// balanced lists of a whole problem), or, without lists, segments lo + b,
// lo + b + grid, ... below hi (a band of output rows).  It travels with the
// tensor maps and the problem in the launch's parameters, so that a CTA's first
// copy waits for one load from global memory (its first segment).
struct SegOrder {
    int lists, lo, hi;
    int begin[CA3DMM_DGEMM_SEG_CTAS + 1];
};

struct SegCursor {
    int pos, end, step, kt, kt1, m0, n0;
    bool valid;
};

template <bool AK, int TBN>
__global__ void __launch_bounds__(THREADS, 1)
dgemm_dmma_segments(const __grid_constant__ CUtensorMap map_a,
                    const __grid_constant__ CUtensorMap map_b, const __grid_constant__ DProb prob,
                    const __grid_constant__ SegOrder order,
                    const ca3dmm_dgemm_seg_t *__restrict__ segs, int uncut,
                    double2 *__restrict__ partials, int *__restrict__ counters, int *status,
                    unsigned long long limit_ns)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    using T = DTile<TBN>;
    constexpr int STAGES = T::STAGES, STAGE_BYTES = T::STAGE_BYTES, MI = T::MI;
    constexpr uint32_t TOTAL_COLS = 2 * 32 * MI;      // two warps per TMEM lane quarter
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + STAGES * STAGE_BYTES);
    uint64_t *empty = full + STAGES;
    __shared__ volatile int abort_flag;
    __shared__ uint64_t fix_bar[2];                   // partial written; the counter's answer
    __shared__ volatile int last_part;
    __shared__ uint32_t tmem_slot;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool producer = threadIdx.x == 0;
    if (producer) {
        tmap_prefetch(&map_a);
        tmap_prefetch(&map_b);
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], CONSUMER_WARPS);
        }
        mbar_init(&fix_bar[0], CONSUMER_WARPS);
        mbar_init(&fix_bar[1], 1);
        abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&tmem_slot)),
                     "r"(TOTAL_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t total = tmem_slot + ((uint32_t) ((warp & 3) * 32) << 16) +
                           (uint32_t) ((warp >> 2) * 32 * MI);

    const int first = order.lists ? order.begin[blockIdx.x] : order.lo + (int) blockIdx.x;
    const int end = order.lists ? order.begin[blockIdx.x + 1] : order.hi;
    const int step = order.lists ? 1 : (int) gridDim.x;

    // thread 0's cursor over the loads, in shared memory: in registers every
    // thread would hold it, and the K-major form spilled
    __shared__ SegCursor lc;
    uint32_t issued = 0;
    auto open_seg = [&]() {
        lc.valid = lc.pos < end;
        if (!lc.valid) return;
        const ca3dmm_dgemm_seg_t &g = segs[lc.pos];
        lc.kt = g.kt0;
        lc.kt1 = g.kt1;
        lc.m0 = g.tm * BM;
        lc.n0 = g.tn * TBN;
    };
    // Issue load number `issued` at the cursor (producer thread only).
    auto issue_one = [&]() -> bool {
        if (!lc.valid) return true;
        const uint32_t s = issued % STAGES, ph = (issued / STAGES) & 1u;
        if (!mbar_wait_bounded(&empty[s], ph ^ 1u, &abort_flag, status,
                               CA3DMM_DEV_TIMEOUT_PRODUCE, limit_ns))
            return false;
        const CUtensorMap *ta = &map_a, *tb = &map_b;
        uint8_t *sA = smem + s * STAGE_BYTES;
        uint8_t *sB = sA + A_BYTES;
        mbar_arrive_expect_tx(&full[s], STAGE_BYTES);
        if (AK) {
            tma_load_2d(sA, ta, lc.kt * BK, lc.m0, &full[s]);
        } else {
#pragma unroll
            for (int j = 0; j < BM / 16; ++j)
                tma_load_2d(sA + j * 2048, ta, lc.m0 + 16 * j, lc.kt * BK, &full[s]);
        }
        tma_load_2d(sB, tb, lc.kt * BK, lc.n0, &full[s]);
        ++issued;
        if (++lc.kt >= lc.kt1) {
            lc.pos += step;
            open_seg();
        }
        return true;
    };
    if (producer) {
        lc.pos = first;
        open_seg();
        for (int s = 0; s < STAGES - 1; ++s)
            if (!issue_one()) break;
    }

    const int g = lane >> 2, t = lane & 3;
    const int wm = warp / T::WN, wn = warp % T::WN;
    uint32_t it = 0;            // loads consumed so far
    uint32_t nfix = 0;          // partial tiles written so far (phase of fix_bar)
    double acc[MI][4][4];
    bool ok = true;

    for (int pos = first; pos < end && ok; pos += step) {
        const ca3dmm_dgemm_seg_t &sg = segs[pos];
        int left = sg.kt1 - sg.kt0;
        int chunk = CA3DMM_DGEMM_CHUNK;
        bool half = left > chunk;                    // the chain of half a chunk is to come
        if (uncut && left > 5 && left < 4 * chunk) {
            const int chains = (left + chunk - 1) / chunk + 1;
            chunk = (left + chains - 1) / chains;
            half = false;
        }
        bool totalled = false;
        for (;;) {
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0;
            int now = min(left, chunk);
            if (half && left <= chunk + chunk / 2) {
                now = chunk / 2;
                half = false;
            }
            ok = k_loop<AK, TBN>(smem, full, empty, now, it, acc, &abort_flag, status, limit_ns,
                                 producer, issue_one, wm, wn, g, t, lane);
            if (!ok) break;
            left -= now;
            if (totalled) {
#pragma unroll
                for (int i = 0; i < MI; ++i) total_add(total + 32 * i, acc[i]);
            }
            if (left <= 0) break;
#pragma unroll
            for (int i = 0; i < MI; ++i) total_store(total + 32 * i, acc[i]);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            totalled = true;
        }
        if (!ok) break;

        const int nparts = sg.nparts;
        if (nparts > 1) {
            // words of a partial tile: (m16 tile, n8 tile, row half) outermost, then the thread
            constexpr int PART = MI * 8 * THREADS;           // double2 of one partial tile
            double2 *mine = partials + (long long) (sg.slot0 + sg.part) * PART + threadIdx.x;
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    __stcg(mine + (i * 8 + j * 2) * THREADS, make_double2(acc[i][j][0], acc[i][j][1]));
                    __stcg(mine + (i * 8 + j * 2 + 1) * THREADS,
                           make_double2(acc[i][j][2], acc[i][j][3]));
                }
            __threadfence();
            __syncwarp();
            if (lane == 0) mbar_arrive(&fix_bar[0]);
            const uint32_t ph = nfix & 1u;
            ++nfix;
            // (a wait that fails here has raised the abort flag, which ends the next one)
            if (producer && mbar_wait_bounded(&fix_bar[0], ph, &abort_flag, status,
                                              CA3DMM_DEV_TIMEOUT_ACCUM, limit_ns)) {
                const bool last = atomicAdd(counters + sg.counter, 1) == nparts - 1;
                if (last) counters[sg.counter] = 0;      // for the next launch
                __threadfence();
                last_part = last;
                mbar_arrive(&fix_bar[1]);
            }
            ok = mbar_wait_warp(&fix_bar[1], ph, &abort_flag, status, CA3DMM_DEV_TIMEOUT_ACCUM,
                                limit_ns);
            if (!ok) break;
            if (!last_part) continue;
            __threadfence();
            const double2 *part = partials + (long long) sg.slot0 * PART + threadIdx.x;
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const double2 lo = __ldcg(part + (i * 8 + j * 2) * THREADS);
                    const double2 hi = __ldcg(part + (i * 8 + j * 2 + 1) * THREADS);
                    acc[i][j][0] = lo.x; acc[i][j][1] = lo.y;
                    acc[i][j][2] = hi.x; acc[i][j][3] = hi.y;
                }
            for (int q = 1; q < nparts; ++q) {
                part += PART;
#pragma unroll
                for (int i = 0; i < MI; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const double2 lo = __ldcg(part + (i * 8 + j * 2) * THREADS);
                        const double2 hi = __ldcg(part + (i * 8 + j * 2 + 1) * THREADS);
                        acc[i][j][0] += lo.x; acc[i][j][1] += lo.y;
                        acc[i][j][2] += hi.x; acc[i][j][3] += hi.y;
                    }
            }
        }
        const int mb = sg.tm * BM + wm * 16 * MI + 2 * (AK ? sigma_row(g) : g);
        const int nb = sg.tn * TBN + wn * 32 + 8 * t;
        store_tile<MI>(prob, mb, nb, acc);
    }

    if (producer) {
        // as above: no TMA write may land in shared memory after exit
        const uint32_t from = issued > STAGES ? issued - STAGES : 0;
        for (uint32_t L = from; L < issued; ++L) {
            const uint32_t s = L % STAGES, ph = (L / STAGES) & 1u;
            uint64_t t0 = global_timer_ns();
            while (!mbar_try_wait(&full[s], ph)) {
                if (global_timer_ns() - t0 > limit_ns) {
                    atomicCAS(status, 0, CA3DMM_DEV_TIMEOUT_PRODUCE);
                    break;
                }
            }
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_slot),
                     "r"(TOTAL_COLS)
                     : "memory");
    }
}

typedef CUresult (*encode_tiled_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                    const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                    const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                    CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

encode_tiled_fn get_encode()
{
    // resolved once; the initialisation of a function-local static is thread-safe
    static const encode_tiled_fn fn = []() -> encode_tiled_fn {
        cudaDriverEntryPointQueryResult q;
        void *p = nullptr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return nullptr;
        return reinterpret_cast<encode_tiled_fn>(p);
    }();
    return fn;
}

// cuTensorMapEncodeTiled is a driver call: it fails in a host thread that has
// no current context, which a thread that has made no runtime call yet lacks
// (the runtime binds the primary context lazily).  cudaSetDevice binds the
// current device's primary context to the calling thread without waiting on
// any stream.
void bind_device_context()
{
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaSetDevice(dev);
}

}  // namespace

extern "C" int ca3dmm_encode_tmap_2d(void *tmap, int dtype_bytes, const void *base,
                                     unsigned long long dim0, unsigned long long dim1,
                                     unsigned long long stride1_bytes, unsigned box0,
                                     unsigned box1, int swizzle128)
{
    encode_tiled_fn enc = get_encode();
    if (!enc) return CA3DMM_ENODEV;
    if ((reinterpret_cast<uintptr_t>(base) & 15) || (stride1_bytes & 15)) return CA3DMM_EINVAL;
    bind_device_context();
    CUtensorMapDataType dt =
        dtype_bytes == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_UINT8;
    cuuint64_t dims[2] = {dim0, dim1};
    cuuint64_t strides[1] = {stride1_bytes};
    cuuint32_t box[2] = {box0, box1};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(reinterpret_cast<CUtensorMap *>(tmap), dt, 2, const_cast<void *>(base), dims,
                     strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     swizzle128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? CA3DMM_OK : CA3DMM_EINVAL;
}

extern "C" int ca3dmm_encode_tmap_u8(void *tmap, int rank, const void *base,
                                     const unsigned long long *dims,
                                     const unsigned long long *strides_bytes,
                                     const unsigned *box)
{
    encode_tiled_fn enc = get_encode();
    if (!enc) return CA3DMM_ENODEV;
    if (rank < 1 || rank > 5 || (reinterpret_cast<uintptr_t>(base) & 15)) return CA3DMM_EINVAL;
    bind_device_context();
    cuuint64_t d[5], st[4];
    cuuint32_t bx[5], es[5];
    for (int i = 0; i < rank; ++i) {
        d[i] = dims[i];
        bx[i] = box[i];
        es[i] = 1;
        if (i > 0) {
            if (strides_bytes[i - 1] & 15) return CA3DMM_EINVAL;
            st[i - 1] = strides_bytes[i - 1];
        }
    }
    CUresult r = enc(reinterpret_cast<CUtensorMap *>(tmap), CU_TENSOR_MAP_DATA_TYPE_UINT8,
                     (cuuint32_t) rank, const_cast<void *>(base), d, st, bx, es,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? CA3DMM_OK : CA3DMM_EINVAL;
}

extern "C" size_t ca3dmm_dgemm_plan_bytes(int nprob)
{
    return (size_t) nprob * 2 * sizeof(CUtensorMap) + (size_t) nprob * sizeof(DProb);
}

extern "C" int ca3dmm_dgemm_plan_encode(const ca3dmm_dgemm_desc_t *probs, int nprob,
                                        void *host_plan, int *total_tiles)
{
    return ca3dmm_dgemm_plan_encode_tn(probs, nprob, host_plan, total_tiles, 128);
}

extern "C" int ca3dmm_dgemm_plan_encode_tn(const ca3dmm_dgemm_desc_t *probs, int nprob,
                                           void *host_plan, int *total_tiles, int tile_n)
{
    if (tile_n != 128 && tile_n != 64) return CA3DMM_EINVAL;
    CUtensorMap *tm = reinterpret_cast<CUtensorMap *>(host_plan);
    DProb *dp = reinterpret_cast<DProb *>(tm + 2 * nprob);
    int tiles = 0;
    for (int i = 0; i < nprob; ++i) {
        const ca3dmm_dgemm_desc_t &q = probs[i];
        if (q.m < 0 || q.n < 0 || q.k < 0) return CA3DMM_EINVAL;
        if ((q.a_kmajor != 0) != (probs[0].a_kmajor != 0)) return CA3DMM_EINVAL;
        if ((q.lda & 1) || (q.ldb & 1) || q.lda < (q.a_kmajor ? q.k : q.m) || q.ldb < q.k)
            return CA3DMM_EINVAL;
        memset(&tm[2 * i], 0, 2 * sizeof(CUtensorMap));
        if (q.m > 0 && q.n > 0 && q.k > 0) {
            int r = q.a_kmajor
                        ? ca3dmm_encode_tmap_2d(&tm[2 * i], 8, q.A, (unsigned long long) q.k,
                                                (unsigned long long) q.m,
                                                (unsigned long long) q.lda * 8, 16, BM, 1)
                        : ca3dmm_encode_tmap_2d(&tm[2 * i], 8, q.A, (unsigned long long) q.m,
                                                (unsigned long long) q.k,
                                                (unsigned long long) q.lda * 8, 16, 16, 1);
            if (r) return r;
            r = ca3dmm_encode_tmap_2d(&tm[2 * i + 1], 8, q.B, (unsigned long long) q.k,
                                      (unsigned long long) q.n, (unsigned long long) q.ldb * 8,
                                      16, (unsigned) tile_n, 1);
            if (r) return r;
        }
        DProb &d = dp[i];
        memset(&d, 0, sizeof(d));
        d.C = q.C;
        d.ldc = q.ldc;
        d.m = q.m; d.n = q.n; d.k = q.k;
        d.alpha = q.alpha; d.beta = q.beta;
        // k == 0 still needs the beta-scaling pass; give it one tile per block
        // through the normal path (ktiles == 0 -> acc stays 0).
        d.tiles_m = (q.m > 0 && q.n > 0) ? (q.m + BM - 1) / BM : 0;
        d.tiles_n = (q.m > 0 && q.n > 0) ? (q.n + tile_n - 1) / tile_n : 0;
        d.tile_begin = tiles;
        d.vec_ok = ((reinterpret_cast<uintptr_t>(q.C) & 15) == 0) && ((q.ldc & 1) == 0);
        d.raster = q.raster > 0 ? q.raster : GROUP_M;
        tiles += d.tiles_m * d.tiles_n;
    }
    *total_tiles = tiles;
    return CA3DMM_OK;
}

extern "C" int ca3dmm_dgemm_launch(const void *dev_plan, int nprob, int total_tiles, int a_kmajor,
                                   int *dev_status, double timeout_s, cudaStream_t stream)
{
    return ca3dmm_dgemm_launch_tn(dev_plan, nprob, total_tiles, a_kmajor, dev_status, timeout_s,
                                  stream, 128);
}

extern "C" int ca3dmm_dgemm_launch_tn(const void *dev_plan, int nprob, int total_tiles,
                                      int a_kmajor, int *dev_status, double timeout_s,
                                      cudaStream_t stream, int tile_n)
{
    ca3dmm_tile_ranges_t rg;
    memset(&rg, 0, sizeof(rg));
    rg.n = 1;
    rg.len[0] = total_tiles;
    return ca3dmm_dgemm_launch_ranges_tn(dev_plan, nprob, &rg, a_kmajor, dev_status, timeout_s,
                                         stream, tile_n);
}

extern "C" int ca3dmm_dgemm_launch_ranges(const void *dev_plan, int nprob,
                                          const ca3dmm_tile_ranges_t *ranges, int a_kmajor,
                                          int *dev_status, double timeout_s, cudaStream_t stream)
{
    return ca3dmm_dgemm_launch_ranges_tn(dev_plan, nprob, ranges, a_kmajor, dev_status, timeout_s,
                                         stream, 128);
}

namespace {
// the shared-memory limit of one instantiation, raised once per device (a bit
// per device ordinal; two threads may both set it, which is harmless)
template <bool AK, int TBN>
cudaError_t dgemm_attr_once()
{
    static std::atomic<unsigned long long> done{0};
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
    if (!bit || !(done.load(std::memory_order_acquire) & bit)) {
        err = cudaFuncSetAttribute(dgemm_dmma_grouped<AK, TBN>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int) DTile<TBN>::SMEM_BYTES);
        if (err != cudaSuccess) return err;
        done.fetch_or(bit, std::memory_order_release);
    }
    return cudaSuccess;
}

template <bool AK, int TBN>
cudaError_t dgemm_launch_one(int grid, const CUtensorMap *tm, const DProb *dp, int nprob,
                             const ca3dmm_tile_ranges_t &rg, int total_tiles, int *status,
                             unsigned long long limit, cudaStream_t stream)
{
    cudaError_t err = dgemm_attr_once<AK, TBN>();
    if (err != cudaSuccess) return err;
    dgemm_dmma_grouped<AK, TBN><<<grid, THREADS, DTile<TBN>::SMEM_BYTES, stream>>>(
        tm, dp, nprob, rg, total_tiles, status, limit);
    return cudaGetLastError();
}
}  // namespace

extern "C" int ca3dmm_dgemm_launch_ranges_tn(const void *dev_plan, int nprob,
                                             const ca3dmm_tile_ranges_t *ranges, int a_kmajor,
                                             int *dev_status, double timeout_s,
                                             cudaStream_t stream, int tile_n)
{
    if (!ranges || ranges->n < 0 || ranges->n > CA3DMM_MAX_RANGES) return CA3DMM_EINVAL;
    if (tile_n != 128 && tile_n != 64) return CA3DMM_EINVAL;
    const int total_tiles = range_total(*ranges);
    if (total_tiles <= 0) return CA3DMM_OK;
    const CUtensorMap *tm = reinterpret_cast<const CUtensorMap *>(dev_plan);
    const DProb *dp = reinterpret_cast<const DProb *>(tm + 2 * nprob);
    int grid = ca3dmm_device_sm_count();
    if (grid > total_tiles) grid = total_tiles;
    const unsigned long long limit = (unsigned long long) (timeout_s * 1e9);
    cudaError_t err;
    if (tile_n == 128)
        err = a_kmajor ? dgemm_launch_one<true, 128>(grid, tm, dp, nprob, *ranges, total_tiles,
                                                      dev_status, limit, stream)
                       : dgemm_launch_one<false, 128>(grid, tm, dp, nprob, *ranges, total_tiles,
                                                       dev_status, limit, stream);
    else
        err = a_kmajor ? dgemm_launch_one<true, 64>(grid, tm, dp, nprob, *ranges, total_tiles,
                                                     dev_status, limit, stream)
                       : dgemm_launch_one<false, 64>(grid, tm, dp, nprob, *ranges, total_tiles,
                                                      dev_status, limit, stream);
    CA3DMM_CUDA_TRY(err);
    ca3dmm_note_launch(1);
    return CA3DMM_OK;
}

// ------------------------------------------------------------------ k segments, host side
// The k segments of an m x n x k product, in tiles of 128 rows x 128 columns
// taken in bands of 8 tile rows (the GEMM's raster order).  `grid` CTAs share
// the tiles' 16-k blocks equally: after `whole` rounds of whole tiles (one tile
// per CTA and round) the blocks of the remaining tiles are cut at multiples of
// their number / grid.  The cuts depend on (m, n, k) alone, not on the tile
// width, the raster or the operands' layout, and neither do the results.
//
// When (all in units of a 16-k block of one tile, 2.2 us of an SM): whole tiles
// take ceil(T / 148) K.  Cut tiles take T K / grid and, for writing the partials
// and adding them up, from 2 (CTAs inside one tile each) to 7 (every CTA between two
// tiles): fitted to 530 shapes of 1 to 2368 tiles and 2 to 1024 blocks, where the
// choice is within 7 % of the better one and 0.06 % on average (with 1.9 in place of
// 2 to 7 it lost up to 16 %, 1408 x 1408 x 256 took 78 us and now takes 68).  At 1000^3
// (T = 64, K = 63) 31 blocks against 63: a call takes 101 us, 194 in whole tiles.
// Products of four rounds or more that equal shares would not shorten by 2 % stay
// with the grouped kernel (one chain over k, no restarts).  Whole tiles run here
// with restarts, those of less than 1024 k in one chain more than they must and all
// of one length, as cut tiles have on average: the errors do not grow where the
// tiles are left whole (1408 x 1408 x 256 in one chain 1.87e-16 of |A||B| rms, cut
// 1.47e-16, in two 1.34e-16; without the restarts long products are 3 to 5 % faster
// and their errors twice as large).
// A product of few blocks is not spread over all SMs: the partials read back by
// the last CTA of a tile grow with the parts, so the number of CTAs is at most
// sqrt(2.5 T T K).  From k = 512 on a share is at least one chunk: chains of 256 k
// keep the error of this path, which the accuracy guard of the tuner and the
// split-precision modes are held against, close below that of the sub-slabs of 512
// k and more (in shares of 187 k a 768^3 product is off by 4.0e-16, less than the
// seven INT8 slices that are to match it, 4.5e-16).  The price at 768^3: 16 blocks
// per CTA instead of 12.
namespace {
constexpr int SEG_SMS = CA3DMM_DGEMM_SEG_CTAS, SEG_RASTER = 8;

struct SegShape {
    long long T, K;              // 128 x 128 tiles, 16-k blocks of a tile
    int tiles_m, tiles_n, grid;
    long long whole;             // rounds of whole tiles before the cut ones (-1: nothing is cut)
};

bool seg_shape(int m, int n, int k, SegShape &s)
{
    if (m <= 0 || n <= 0 || k <= 0) return false;
    s.tiles_m = (m + 127) / 128;
    s.tiles_n = (n + 127) / 128;
    s.T = (long long) s.tiles_m * s.tiles_n;
    s.K = ((long long) k + BK - 1) / BK;
    if (s.T > CA3DMM_DGEMM_SEG_TILES) return false;
    const double dp = (double) ((s.T + SEG_SMS - 1) / SEG_SMS) * (double) s.K;
    double g = std::sqrt(2.5 * (double) s.T * (double) s.T * (double) s.K);
    if (g > SEG_SMS) g = SEG_SMS;
    if (g > (double) (s.T * s.K)) g = (double) (s.T * s.K);
    if (s.K >= 2 * CA3DMM_DGEMM_CHUNK && g > (double) (s.T * s.K / CA3DMM_DGEMM_CHUNK))
        g = (double) (s.T * s.K / CA3DMM_DGEMM_CHUNK);
    s.grid = g < 1.0 ? 1 : (int) g;
    const double share = (double) s.T * (double) s.K / s.grid;
    if (s.T >= 4 * SEG_SMS && share + 1.9 >= 0.98 * dp) return false;
    const double spread = s.T < s.grid ? (double) s.T / s.grid : 1.0;
    if (share + 2.0 + 5.0 * spread < dp) {
        s.whole = s.T / s.grid > 1 ? s.T / s.grid - 1 : 0;
    } else {
        s.whole = -1;
        s.grid = s.T < SEG_SMS ? (int) s.T : SEG_SMS;
    }
    return true;
}

// Cut points of the tiles after the whole ones, in blocks; one within 1/16 of a
// share (or one block) of a tile's edge moves there, which saves a partial.
// Returns the number of whole tiles.
long long seg_cuts(const SegShape &s, long long (&cut)[SEG_SMS + 1])
{
    const int G = s.grid;
    const long long dp = s.whole < 0 ? s.T : s.whole * G;
    const long long U = (s.T - dp) * s.K;
    const long long slack = U / G / 16 > 1 ? U / G / 16 : 1;
    for (int c = 0; c <= G; ++c) {
        long long u = U > 0 ? U * c / G : 0;
        if (c > 0 && c < G) {
            const long long r = u % s.K;
            if (r <= slack && r < s.K - r) u -= r;
            else if (s.K - r <= slack) u += s.K - r;
            if (u < cut[c - 1]) u = cut[c - 1];
        }
        cut[c] = u;
    }
    return dp;
}

void seg_tile(const SegShape &s, long long tile, int &tm, int &tn)
{
    const long long per = (long long) SEG_RASTER * s.tiles_n, b = tile / per, r = tile % per;
    const int first = (int) b * SEG_RASTER;
    const int rows = s.tiles_m - first < SEG_RASTER ? s.tiles_m - first : SEG_RASTER;
    tm = first + (int) (r % rows);
    tn = (int) (r / rows);
}
}  // namespace

extern "C" int ca3dmm_dgemm_segments_max(int m, int n, int k)
{
    SegShape s;
    if (!seg_shape(m, n, k, s)) return 0;
    return (int) (2 * (s.T + s.grid));
}

extern "C" size_t ca3dmm_dgemm_segments_ws_bytes(int m, int n, int k)
{
    SegShape s;
    if (!seg_shape(m, n, k, s) || s.whole < 0) return 0;
    // every cut inside a tile adds a partial, the first of a tile's two
    long long cut[SEG_SMS + 1], tile = -1, last = 0, slots = 0;
    seg_cuts(s, cut);
    for (int c = 1; c < s.grid; ++c) {
        if (cut[c] % s.K == 0 || cut[c] == last) continue;
        last = cut[c];
        slots += last / s.K == tile ? 1 : 2;
        tile = last / s.K;
    }
    return (size_t) slots * BM * 128 * sizeof(double);
}

extern "C" int ca3dmm_dgemm_segments(int m, int n, int k, int tile_n, ca3dmm_dgemm_seg_t *segs,
                                     int *order, int *cta_begin, int *nseg, int *grid,
                                     int *ncounter)
{
    SegShape s;
    *nseg = *grid = *ncounter = 0;
    if (!seg_shape(m, n, k, s) || (tile_n != 128 && tile_n != 64)) return CA3DMM_EINVAL;
    const int G = s.grid;
    int ns = 0, nc = 0, slots = 0;
    long long cut[SEG_SMS + 1];
    const long long dp = seg_cuts(s, cut);                      // whole tiles
    // segments in tile order, each with the CTA that runs it
    int *who = static_cast<int *>(malloc(sizeof(int) * (size_t) (2 * (s.T + G) + 1)));
    if (!who) return CA3DMM_ENOMEM;
    int c = 0;                                                  // CTA holding block u
    for (long long tile = 0; tile < s.T; ++tile) {
        int tm, tn;
        seg_tile(s, tile, tm, tn);
        const int halves = tile_n == 128 ? 1 : (n - tn * 128 > 64 ? 2 : 1);
        long long u0 = 0;
        if (tile >= dp) {
            u0 = (tile - dp) * s.K;
            while (c + 1 < G && cut[c + 1] <= u0) ++c;
        }
        for (int h = 0; h < halves; ++h) {
            int q = c, part = 0;
            long long from = 0;
            do {
                ca3dmm_dgemm_seg_t &g = segs[ns];
                long long to = s.K;
                if (tile >= dp) {
                    // skip CTAs left empty by moved cut points
                    while (q + 1 < G && cut[q + 1] <= u0 + from) ++q;
                    if (q + 1 < G && cut[q + 1] < u0 + s.K) to = cut[q + 1] - u0;
                }
                g.tm = tm;
                g.tn = tile_n == 128 ? tn : 2 * tn + h;
                g.kt0 = (int) from;
                g.kt1 = (int) to;
                g.part = part++;
                g.nparts = 0;
                g.slot0 = 0;
                g.counter = 0;
                who[ns++] = tile < dp ? (int) (tile % G) : q;
                from = to;
            } while (from < s.K);
            for (int i = 0; i < part; ++i) {
                ca3dmm_dgemm_seg_t &g = segs[ns - part + i];
                g.nparts = part;
                g.slot0 = part > 1 ? slots : 0;
                g.counter = part > 1 ? nc : 0;
            }
            if (part > 1) { slots += part; ++nc; }
        }
    }
    // per-CTA lists, in tile order
    for (int b = 0; b <= G; ++b) cta_begin[b] = 0;
    for (int i = 0; i < ns; ++i) ++cta_begin[who[i] + 1];
    for (int b = 0; b < G; ++b) cta_begin[b + 1] += cta_begin[b];
    int *at = static_cast<int *>(malloc(sizeof(int) * (size_t) (G + 1)));
    if (!at) { free(who); return CA3DMM_ENOMEM; }
    memcpy(at, cta_begin, sizeof(int) * (size_t) G);
    for (int i = 0; i < ns; ++i) order[at[who[i]]++] = i;
    free(at);
    free(who);
    *nseg = ns;
    *grid = G;
    *ncounter = nc;
    return CA3DMM_OK;
}

namespace {
template <bool AK, int TBN>
cudaError_t seg_launch_one(int grid, const CUtensorMap *tm, const DProb &prob, const SegOrder &o,
                           const ca3dmm_dgemm_seg_t *segs, int uncut, double2 *partials,
                           int *counters, int *status, unsigned long long limit,
                           cudaStream_t stream)
{
    static std::atomic<unsigned long long> done{0};      // as dgemm_attr_once
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
    if (!bit || !(done.load(std::memory_order_acquire) & bit)) {
        err = cudaFuncSetAttribute(dgemm_dmma_segments<AK, TBN>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int) DTile<TBN>::SMEM_BYTES);
        if (err != cudaSuccess) return err;
        done.fetch_or(bit, std::memory_order_release);
    }
    dgemm_dmma_segments<AK, TBN><<<grid, THREADS, DTile<TBN>::SMEM_BYTES, stream>>>(
        tm[0], tm[1], prob, o, segs, uncut, partials, counters, status, limit);
    return cudaGetLastError();
}
}  // namespace

extern "C" int ca3dmm_dgemm_launch_segments(const void *host_plan, int nprob,
                                            const ca3dmm_dgemm_seg_t *dev_segs,
                                            const int *cta_begin, int lo, int hi, int grid,
                                            int a_kmajor, void *partials, int *counters,
                                            int *dev_status, double timeout_s, cudaStream_t stream,
                                            int tile_n)
{
    if (tile_n != 128 && tile_n != 64) return CA3DMM_EINVAL;
    if (hi <= lo) return CA3DMM_OK;
    const CUtensorMap *tm = reinterpret_cast<const CUtensorMap *>(host_plan);
    const DProb &prob = *reinterpret_cast<const DProb *>(tm + 2 * nprob);
    SegOrder o;
    memset(&o, 0, sizeof(o));
    o.lists = cta_begin != nullptr;
    o.lo = lo;
    o.hi = hi;
    if (cta_begin) {
        if (grid < 1 || grid > CA3DMM_DGEMM_SEG_CTAS) return CA3DMM_EINVAL;
        memcpy(o.begin, cta_begin, sizeof(int) * (size_t) (grid + 1));
    } else {
        grid = ca3dmm_device_sm_count();
        if (grid > hi - lo) grid = hi - lo;
    }
    SegShape s;
    if (!seg_shape(prob.m, prob.n, prob.k, s)) return CA3DMM_EINVAL;
    const unsigned long long limit = (unsigned long long) (timeout_s * 1e9);
    double2 *ws = static_cast<double2 *>(partials);
    const int uncut = s.whole < 0;
    cudaError_t err;
    if (tile_n == 128)
        err = a_kmajor ? seg_launch_one<true, 128>(grid, tm, prob, o, dev_segs, uncut, ws, counters,
                                                   dev_status, limit, stream)
                       : seg_launch_one<false, 128>(grid, tm, prob, o, dev_segs, uncut, ws, counters,
                                                    dev_status, limit, stream);
    else
        err = a_kmajor ? seg_launch_one<true, 64>(grid, tm, prob, o, dev_segs, uncut, ws, counters,
                                                  dev_status, limit, stream)
                       : seg_launch_one<false, 64>(grid, tm, prob, o, dev_segs, uncut, ws, counters,
                                                   dev_status, limit, stream);
    CA3DMM_CUDA_TRY(err);
    ca3dmm_note_launch(1);
    return CA3DMM_OK;
}

extern "C" int ca3dmm_device_sm_count(void)
{
    static std::atomic<int> sms[64];        // zero-initialised (static storage)
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    int v = sms[dev].load(std::memory_order_relaxed);
    if (!v) {
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0)
            v = 148;
        sms[dev].store(v, std::memory_order_relaxed);
    }
    return v;
}
