// Redistribution kernels of the virtual process grid, HBM-bound:
//   * batched block pack (copy or transpose) of column-major matrices --
//     the on-device form of mat_redist's pack -> alltoallv -> unpack
//     (src/mat_redist.c:327-348, :395-416) fused with the operand transpose
//     the reference does with cublasDgeam (src/ca3dmm.c:1036-1058);
//   * the kp-slab FP64 reduction -- the on-device form of the C
//     reduce-scatter with mpi_op_omp_sum (src/ca3dmm.c:1287-1343,
//     src/mpi_op_omp.c:6-23), summing slabs in rank order.
#include <atomic>
#include <cstring>
#include <cuda.h>
#include <cuda_runtime.h>
#include "k_common.cuh"
#include "ca3dmm_kernels.h"

namespace {

constexpr int PT = 64;   // pack tile edge
// (n + 63 may not fit)
__host__ __device__ constexpr int pack_tiles_of(int n) { return (n - 1) / PT + 1; }

__device__ __forceinline__ int find_desc(const ca3dmm_pack_desc_t *d, int n, int tile)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (d[mid].tile_begin <= tile) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Persistent over the flat list of 64 x 64 tiles of every descriptor.
// Copy: thread -> (row, 16 columns), reads and writes run down the columns.
// Transpose: through a padded shared tile; reads run along the source's
// contiguous index, writes along the destination's.
__global__ void __launch_bounds__(256, 3)
pack_kernel(const double *__restrict__ src_base, double *__restrict__ dst_base,
            const ca3dmm_pack_desc_t *__restrict__ descs, int ndesc, int total_tiles)
{
    __shared__ double tile[PT][PT + 1];
    for (int t = blockIdx.x; t < total_tiles; t += gridDim.x) {
        const ca3dmm_pack_desc_t d = descs[find_desc(descs, ndesc, t)];
        const int local = t - d.tile_begin;
        const int tx = pack_tiles_of(d.rows);
        const int r0 = (local % tx) * PT, c0 = (local / tx) * PT;
        const double *src = reinterpret_cast<const double *>(
            reinterpret_cast<uintptr_t>(src_base) + (uintptr_t) d.src_off * sizeof(double));
        double *dst = reinterpret_cast<double *>(reinterpret_cast<uintptr_t>(dst_base) +
                                                 (uintptr_t) d.dst_off * sizeof(double));
        if (!d.trans) {
            const int r = r0 + (threadIdx.x & 63), cb = c0 + (threadIdx.x >> 6) * 16;
            if (r < d.rows) {
                double v[16];
#pragma unroll
                for (int c = 0; c < 16; ++c)
                    if (cb + c < d.cols) v[c] = __ldg(src + r + (long long) (cb + c) * d.lds);
#pragma unroll
                for (int c = 0; c < 16; ++c)
                    if (cb + c < d.cols) dst[r + (long long) (cb + c) * d.ldd] = v[c];
            }
            continue;
        }
        // dst (rows x cols) = transpose of the source block (cols x rows); the
        // 16 loads of a thread are all in flight before the shared stores
        double v[PT * PT / 256];
#pragma unroll
        for (int i = 0; i < PT * PT / 256; ++i) {
            const int e = threadIdx.x + 256 * i;
            const int c = c0 + (e & 63), r = r0 + (e >> 6);
            v[i] = (c < d.cols && r < d.rows) ? __ldg(src + c + (long long) r * d.lds) : 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < PT * PT / 256; ++i) {
            const int e = threadIdx.x + 256 * i;
            tile[e >> 6][e & 63] = v[i];
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < PT * PT / 256; ++i) {
            const int e = threadIdx.x + 256 * i;
            const int r = r0 + (e & 63), c = c0 + (e >> 6);
            if (r < d.rows && c < d.cols) dst[r + (long long) c * d.ldd] = tile[e & 63][e >> 6];
        }
    }
}

// Transposing pack staged through shared memory by TMA: tiles of 64
// destination rows x 64 destination columns arrive as four 16 x 64 boxes of
// the source (16 contiguous doubles = one 128-byte box row, so 512
// contiguous source bytes per row and tile) with the 128-byte swizzle,
// TT_STAGES tiles ahead of the threads that write them out.  A thread reads
// 16-byte chunks (two destination columns of one row): 32 threads of
// consecutive rows hit eight distinct swizzled chunks, the minimum four
// wavefronts; the writes run down the destination columns.
constexpr int TT_R = 64, TT_BOX = 16, TT_NBOX = 4, TT_C = TT_BOX * TT_NBOX, TT_STAGES = 4;
constexpr int TT_BOX_BYTES = TT_R * TT_BOX * (int) sizeof(double);   // 8 KB
constexpr int TT_BYTES = TT_BOX_BYTES * TT_NBOX;                       // 32 KB
constexpr int TT_SMEM = TT_STAGES * TT_BYTES + 1024;

__device__ __forceinline__ void tt_tile(const ca3dmm_pack_desc_t &d, int t, int &r0, int &c0)
{
    const int local = t - d.tile_begin, tr = (d.rows + TT_R - 1) / TT_R;
    r0 = (local % tr) * TT_R;
    c0 = (local / tr) * TT_C;
}

__global__ void __launch_bounds__(256)
pack_transpose_tma_kernel(const CUtensorMap *__restrict__ tmaps,
                          const ca3dmm_pack_desc_t *__restrict__ descs, int ndesc, int total_tiles,
                          double *__restrict__ dst_base, int *status, unsigned long long limit_ns)
{
    extern __shared__ unsigned char tt_raw[];
    unsigned char *sm = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(tt_raw) + 1023) & ~uintptr_t(1023));
    __shared__ uint64_t full[TT_STAGES];
    __shared__ volatile int abort_flag;
    if (threadIdx.x == 0) {
        for (int s = 0; s < TT_STAGES; ++s) mbar_init(&full[s], 1);
        abort_flag = 0;
        fence_barrier_init();
    }
    __syncthreads();
    const int mine = blockIdx.x < total_tiles ? (total_tiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;
    int issued = 0;
    auto issue = [&](int i) {
        const int t = blockIdx.x + i * gridDim.x;
        const int j = find_desc(descs, ndesc, t);
        int r0, c0;
        tt_tile(descs[j], t, r0, c0);
        tmap_acquire(tmaps + j);
        const int s = i % TT_STAGES;
        mbar_arrive_expect_tx(&full[s], TT_BYTES);
#pragma unroll
        for (int b = 0; b < TT_NBOX; ++b)
            tma_load_2d(sm + s * TT_BYTES + b * TT_BOX_BYTES, tmaps + j, c0 + b * TT_BOX, r0, &full[s]);
    };
    if (threadIdx.x == 0)
        for (; issued < mine && issued < TT_STAGES; ++issued) issue(issued);
    const int r = threadIdx.x & (TT_R - 1), q0 = threadIdx.x >> 6;
    bool ok = true;
    for (int i = 0; i < mine && ok; ++i) {
        const int s = i % TT_STAGES;
        if (!mbar_wait_warp(&full[s], (uint32_t) (i / TT_STAGES) & 1u, &abort_flag, status,
                            CA3DMM_DEV_TIMEOUT_CONSUME, limit_ns)) {
            ok = false;
            break;
        }
        const int t = blockIdx.x + i * gridDim.x;
        const ca3dmm_pack_desc_t d = descs[find_desc(descs, ndesc, t)];
        int r0, c0;
        tt_tile(d, t, r0, c0);
        double *dst = reinterpret_cast<double *>(reinterpret_cast<uintptr_t>(dst_base) +
                                                 (uintptr_t) d.dst_off * sizeof(double));
        const unsigned char *row = sm + s * TT_BYTES + r * 128;
#pragma unroll
        for (int h = 0; h < TT_C / 8; ++h) {
            const int q = q0 + 4 * h;                       // chunk: columns 2q, 2q + 1
            const double2 v = *reinterpret_cast<const double2 *>(
                row + (q >> 3) * TT_BOX_BYTES + (((q & 7) ^ (r & 7)) << 4));
            const int gr = r0 + r, gc = c0 + 2 * q;
            if (gr < d.rows) {
                if (gc < d.cols) dst[gr + (long long) gc * d.ldd] = v.x;
                if (gc + 1 < d.cols) dst[gr + (long long) (gc + 1) * d.ldd] = v.y;
            }
        }
        __syncthreads();                                     // stage s read by every thread
        if (threadIdx.x == 0 && issued < mine) issue(issued++);
    }
    if (threadIdx.x == 0 && !ok) {
        // let the copies this CTA issued land before its shared memory is released
        for (int i = 0; i < issued; ++i) {
            const uint64_t t0 = global_timer_ns();
            while (!mbar_try_wait(&full[i % TT_STAGES], (uint32_t) (i / TT_STAGES) & 1u))
                if (global_timer_ns() - t0 > limit_ns) break;
        }
    }
}

// out = sum of nslab slabs, column-major, 2 doubles per thread when aligned.
__global__ void __launch_bounds__(256)
reduce_slabs_kernel(const double *__restrict__ slab, long long slab_stride, long long lds,
                    int nslab, int m, int n, double *__restrict__ out, long long ldo, int vec)
{
    const long long mh = vec ? (m + 1) / 2 : m;
    const long long total = mh * n;
    for (long long idx = blockIdx.x * (long long) blockDim.x + threadIdx.x; idx < total;
         idx += (long long) gridDim.x * blockDim.x) {
        const long long j = idx / mh;
        const long long i = (idx - j * mh) * (vec ? 2 : 1);
        if (vec && i + 1 < m) {
            const double *p = slab + i + j * lds;
            double2 s = *reinterpret_cast<const double2 *>(p);
            for (int q = 1; q < nslab; ++q) {
                double2 v = *reinterpret_cast<const double2 *>(p + q * slab_stride);
                s.x += v.x;
                s.y += v.y;
            }
            *reinterpret_cast<double2 *>(out + i + j * ldo) = s;
        } else {
            const double *p = slab + i + j * lds;
            double s = p[0];
            for (int q = 1; q < nslab; ++q) s += p[q * slab_stride];
            out[i + j * ldo] = s;
        }
    }
}

}  // namespace

static std::atomic<unsigned long long> g_kernel_launches{0};

extern "C" void ca3dmm_note_launch(int n)
{
    g_kernel_launches.fetch_add((unsigned long long) n, std::memory_order_relaxed);
}

extern "C" unsigned long long ca3dmm_kernel_launches(void)
{
    return g_kernel_launches.load(std::memory_order_relaxed);
}

extern "C" int ca3dmm_pack_tiles(ca3dmm_pack_desc_t *descs, int ndesc)
{
    int tiles = 0;
    for (int j = 0; j < ndesc; ++j) {
        descs[j].tile_begin = tiles;
        if (descs[j].rows > 0 && descs[j].cols > 0)
            tiles += pack_tiles_of(descs[j].rows) * pack_tiles_of(descs[j].cols);
    }
    return tiles;
}

// One block copy with its geometry passed by value (no descriptor in device
// memory): thread (row, 16 columns) of a 128 x 16 tile, the grid's y extent
// walking further column tiles when there are more than 65535 of them.
__global__ void __launch_bounds__(128)
copy_block_kernel(const double *__restrict__ src, long long lds, double *__restrict__ dst,
                  long long ldd, int rows, int cols)
{
    const int r = blockIdx.x * 128 + threadIdx.x;
    if (r >= rows) return;
    for (long long c0 = (long long) blockIdx.y * 16; c0 < cols; c0 += (long long) gridDim.y * 16) {
        double v[16];
#pragma unroll
        for (int c = 0; c < 16; ++c)
            if (c0 + c < cols) v[c] = __ldg(src + r + (c0 + c) * lds);
#pragma unroll
        for (int c = 0; c < 16; ++c)
            if (c0 + c < cols) dst[r + (c0 + c) * ldd] = v[c];
    }
}

// Copies of many blocks with unrelated addresses and leading dimensions, the
// blocks given in the launch's parameters.  HBM bound.  The contiguous runs of a
// block are a few KB and start anywhere (layouts split a matrix into strips of any
// width), so a warp copies whole runs, two at a time with all their loads in
// flight, four per item, up to RUN_E elements of them; its stores cover whole
// lines.  Items go through the blocks in turn, four runs of each, so that the
// blocks that share a destination row fill it at about the same time -- as long as
// the blocks are of about one size: each takes as many turns as the largest.  When
// more than a quarter of the turns would be empty, the items follow the blocks one
// after the other, each block with its own number (one 8000 x 8000 block beside 400
// of 10 x 20, in turn 1657 us, tile copies 314, now 291; 60000 x 8000 beside 300 of
// 1 x 20: 8690, 1357, now 1253).
// 8000 x 8000 from 24 column strips to 4 x 6 blocks (116 pieces, 1.02 GB): 178 us,
// 5.75 TB/s (one piece after the other 199-214; with default loads and stores in
// place of the streaming ones, lines aligned, 373; 64 x 64 tiles from descriptors
// in memory 206).  The call: 241 -> 206 us, with the upload of the descriptors and
// the wait before it gone.
// Runs of up to RUN_NARROW elements are too short for that: two of them in flight are
// less than the memory's latency asks for.  An item takes as many as fill 64 loads of
// every lane, half of them in flight; runs of up to 16 elements lie side by side in
// a warp.  Into 8 row blocks (256 MB each way): 1600000 x 20 in 106 us (385 two runs
// at a time, 167 by tile copies), 1000000 x 32 106 (263, 128), 500000 x 64 105 (164,
// 110), 250000 x 128 106 (119, 109); 400 strips of 20, 64, 100 columns to one block
// 219, 390, 528 us (500, 560, 650; 324, 438, 680).  At 160 and 200 columns both take
// the same time, at 256 whole runs 104 us and this 107; with 16 loads in flight in
// twice the warps 1 to 2 % more, with loads that L1 keeps up to 10 %.
constexpr int RUN_E = 512, RUN_GROUP = 4, RUN_NARROW = 128, RUN_LOADS = 32;
__host__ __device__ inline bool run_narrow(int len) { return len <= RUN_NARROW; }
// narrow: loads per run, and log2 of the lanes that share one
__host__ __device__ inline int run_loads(int len) { return len <= 32 ? 1 : len <= 64 ? 2 : 4; }
__host__ __device__ inline int run_lanes(int len)
{
    return len > 16 ? 5 : len > 8 ? 4 : len > 4 ? 3 : len > 2 ? 2 : len > 1 ? 1 : 0;
}
inline int run_chunks(int len) { return run_narrow(len) ? 1 : (len + 15 + RUN_E - 1) / RUN_E; }
inline int run_group(int len)
{
    return run_narrow(len) ? 2 * (RUN_LOADS / run_loads(len)) << (5 - run_lanes(len)) : RUN_GROUP;
}

struct RunPiece {
    const double *src;
    double *dst;
    int lds, ldd, len, runs;
    int begin, nch, group;           // first item (blocks one after the other), chunks, runs per item
};

template <int CAP>
struct RunPieces {
    RunPiece p[CAP];
};

struct RunItems {
    int npiece, turn, total;         // turn: chunks per block in turn (0: one after the other)
};

struct RunItem {
    int piece, run0, run1, col0;                     // runs [run0, run1), from column col0 on
};

// Item -> what it copies; run0 == run1: nothing (an empty turn).
__host__ __device__ inline RunItem run_item(const RunPiece *p, const RunItems &I, int item)
{
    RunItem o;
    int g, c;
    if (I.turn) {
        const int ic = item / I.turn;
        g = ic / I.npiece;
        o.piece = ic - g * I.npiece;
        c = item - ic * I.turn;
    } else {
        int lo = 0, hi = I.npiece - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (p[mid].begin <= item) lo = mid; else hi = mid - 1;
        }
        o.piece = lo;
        g = (item - p[lo].begin) / p[lo].nch;
        c = (item - p[lo].begin) - g * p[lo].nch;
    }
    const int runs = p[o.piece].runs, group = p[o.piece].group;
    o.col0 = c * RUN_E;
    o.run0 = o.run1 = 0;
    if (c < p[o.piece].nch && (long long) g * group < runs) {
        o.run0 = g * group;
        o.run1 = runs - o.run0 < group ? runs : o.run0 + group;
    }
    return o;
}

// An item of narrow runs, U loads each.
template <int U>
__device__ __forceinline__ void copy_narrow(const RunPiece &d, int run0, int run1, int lane)
{
    const int lg = U == 1 ? run_lanes(d.len) : 5, sub = 32 >> lg;
    const int col = lane & ((1 << lg) - 1);
    const long long ds = (long long) sub * d.lds, dd = (long long) sub * d.ldd;
    const long long first = run0 + (lane >> lg);
    const double *s = d.src + first * d.lds + col;
    double *t = d.dst + first * d.ldd + col;
    int left = (run1 - (int) first + sub - 1) >> (5 - lg);      // runs of this lane
#pragma unroll 1
    for (; left > 0; left -= RUN_LOADS / U) {
        double v[RUN_LOADS];
#pragma unroll
        for (int i = 0; i < RUN_LOADS / U; ++i) {
#pragma unroll
            for (int u = 0; u < U; ++u)
                v[i * U + u] = i < left && col + 32 * u < d.len ? __ldcs(s + 32 * u) : 0.0;
            s += ds;
            asm volatile("" : "+l"(s));              // one address at a time
        }
#pragma unroll
        for (int i = 0; i < RUN_LOADS / U; ++i) {
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (i < left && col + 32 * u < d.len) __stcs(t + 32 * u, v[i * U + u]);
            t += dd;
            asm volatile("" : "+l"(t));
        }
    }
}

template <int CAP>
__global__ void __launch_bounds__(256)
copy_runs_kernel(const __grid_constant__ RunPieces<CAP> P, const RunItems I)
{
    const int lane = threadIdx.x & 31;
    for (int item = blockIdx.x * 8 + (threadIdx.x >> 5); item < I.total; item += gridDim.x * 8) {
        const RunItem w = run_item(P.p, I, item);
        const RunPiece &d = P.p[w.piece];
        const int c0 = w.col0 + lane, r1 = w.run1;
        for (int r = w.run0; r < r1; r += 2) {
            // each run's elements counted from the 128-byte line its destination starts
            // in, so that a warp's store covers whole lines
            const double *s0 = d.src + (long long) r * d.lds;
            double *t0 = d.dst + (long long) r * d.ldd, *t1 = t0 + d.ldd;
            const int e0 = c0 - (int) ((reinterpret_cast<uintptr_t>(t0) >> 3) & 15);
            const int e1 = c0 - (int) ((reinterpret_cast<uintptr_t>(t1) >> 3) & 15);
            const unsigned int len = (unsigned int) d.len, len1 = r + 1 < r1 ? len : 0u;
            s0 += e0;
            const double *s1 = d.src + (long long) (r + 1) * d.lds + e1;
            t0 += e0;
            t1 += e1;
            double v0[RUN_E / 32], v1[RUN_E / 32];
#pragma unroll
            for (int u = 0; u < RUN_E / 32; ++u) {
                if ((unsigned int) (e0 + 32 * u) < len) v0[u] = __ldcs(s0 + 32 * u);
                if ((unsigned int) (e1 + 32 * u) < len1) v1[u] = __ldcs(s1 + 32 * u);
            }
#pragma unroll
            for (int u = 0; u < RUN_E / 32; ++u) {
                if ((unsigned int) (e0 + 32 * u) < len) __stcs(t0 + 32 * u, v0[u]);
                if ((unsigned int) (e1 + 32 * u) < len1) __stcs(t1 + 32 * u, v1[u]);
            }
        }
    }
}

// The same for blocks of narrow runs: a kernel of its own, whose warps need half the
// registers.
template <int CAP>
__global__ void __launch_bounds__(256, 2)
copy_narrow_runs_kernel(const __grid_constant__ RunPieces<CAP> P, const RunItems I)
{
    const int lane = threadIdx.x & 31;
    for (int item = blockIdx.x * 8 + (threadIdx.x >> 5); item < I.total; item += gridDim.x * 8) {
        const RunItem w = run_item(P.p, I, item);
        const RunPiece &d = P.p[w.piece];
        const int loads = run_loads(d.len);
        if (loads == 1) copy_narrow<1>(d, w.run0, w.run1, lane);
        else if (loads == 2) copy_narrow<2>(d, w.run0, w.run1, lane);
        else copy_narrow<4>(d, w.run0, w.run1, lane);
    }
}

// Work items of a launch over these pieces, -1 when their number or the sizes leave
// the kernel's 32-bit counts: it looks up to two chunks past a run's end.
constexpr int RUN_MAX = 0x7fffffff - 4 * RUN_E;
static bool run_plan(const ca3dmm_run_piece_t *pieces, int n, bool narrow, RunPiece *p, RunItems &I)
{
    I = RunItems{0, 0, 0};
    if (n < 0 || n > CA3DMM_MAX_RUN_PIECES) return false;
    long long groups = 0, nch = 0, sum = 0;
    for (int i = 0; i < n; ++i) {
        const ca3dmm_run_piece_t &q = pieces[i];
        if (q.len <= 0 || q.runs <= 0 || run_narrow(q.len) != narrow) continue;
        if (q.len > RUN_MAX || q.runs > RUN_MAX) return false;
        RunPiece &o = p[I.npiece++];
        o.src = q.src; o.dst = q.dst;
        o.lds = q.lds; o.ldd = q.ldd; o.len = q.len; o.runs = q.runs;
        o.nch = run_chunks(q.len);
        o.group = run_group(q.len);
        o.begin = (int) sum;
        const long long g = (q.runs - 1LL) / o.group + 1;
        if (g > groups) groups = g;
        if (o.nch > nch) nch = o.nch;
        sum += g * o.nch;
        if (sum > 1000000000) return false;
    }
    if (sum == 0) return true;
    // (the groups and chunks of one block are at most sum: no overflow before the test)
    const bool turn = (double) groups * I.npiece * (double) nch <= 1.25 * (double) sum;
    I.turn = turn ? (int) nch : 0;
    I.total = (int) (turn ? groups * I.npiece * nch : sum);
    return true;
}

extern "C" long long ca3dmm_copy_runs_items(const ca3dmm_run_piece_t *pieces, int n)
{
    RunPieces<CA3DMM_MAX_RUN_PIECES> P;
    RunItems wide, narrow;
    return run_plan(pieces, n, false, P.p, wide) && run_plan(pieces, n, true, P.p, narrow)
               ? (long long) wide.total + narrow.total : -1;
}

extern "C" int ca3dmm_copy_runs_item(const ca3dmm_run_piece_t *pieces, int n, long long item,
                                     int *out5)
{
    RunPieces<CA3DMM_MAX_RUN_PIECES> P;
    RunItems I;
    if (item < 0 || !run_plan(pieces, n, false, P.p, I)) return CA3DMM_EINVAL;
    const bool narrow = item >= I.total;
    if (narrow) item -= I.total;
    if (!run_plan(pieces, n, narrow, P.p, I) || item >= I.total) return CA3DMM_EINVAL;
    const RunItem w = run_item(P.p, I, (int) item);
    const RunPiece &d = P.p[w.piece];
    out5[0] = 0;
    for (int i = 0, of = 0;; ++i) {
        if (pieces[i].len <= 0 || pieces[i].runs <= 0) continue;
        if (run_narrow(pieces[i].len) == narrow && of++ == w.piece) break;
        ++out5[0];
    }
    out5[1] = w.run0;
    out5[2] = w.run1;
    out5[3] = w.col0;
    out5[4] = d.len + 15 - w.col0 < RUN_E ? d.len + 15 : w.col0 + RUN_E;
    return CA3DMM_OK;
}

template <int CAP>
static cudaError_t copy_runs_launch(const ca3dmm_run_piece_t *pieces, int n, cudaStream_t stream)
{
    RunPieces<CAP> P;
    RunItems I;
    const long long cap = (long long) ca3dmm_device_sm_count() * 64;
    for (int narrow = 0; narrow < 2; ++narrow) {
        if (!run_plan(pieces, n, narrow, P.p, I)) return cudaErrorInvalidValue;
        if (I.total == 0) continue;
        const long long blocks = (I.total + 7LL) / 8;
        const unsigned grid = (unsigned) (blocks < cap ? blocks : cap);
        if (narrow) copy_narrow_runs_kernel<CAP><<<grid, 256, 0, stream>>>(P, I);
        else copy_runs_kernel<CAP><<<grid, 256, 0, stream>>>(P, I);
        ca3dmm_note_launch(1);
    }
    return cudaGetLastError();
}

extern "C" int ca3dmm_copy_runs_launch(const ca3dmm_run_piece_t *pieces, int n, cudaStream_t stream)
{
    if (n < 0 || n > CA3DMM_MAX_RUN_PIECES) return CA3DMM_EINVAL;
    if (n == 0) return CA3DMM_OK;
    // the launch copies its parameters (24 KB at 512 blocks, 2 us): as few as hold them
    CA3DMM_CUDA_TRY(n <= 32    ? copy_runs_launch<32>(pieces, n, stream)
                    : n <= 128 ? copy_runs_launch<128>(pieces, n, stream)
                               : copy_runs_launch<CA3DMM_MAX_RUN_PIECES>(pieces, n, stream));
    return CA3DMM_OK;
}

extern "C" int ca3dmm_copy_block_launch(const double *src, long long lds, double *dst,
                                        long long ldd, int rows, int cols, cudaStream_t stream)
{
    if (rows <= 0 || cols <= 0) return CA3DMM_OK;
    const long long ty = ((long long) cols + 15) / 16;
    dim3 grid((unsigned) ((rows + 127) / 128), (unsigned) (ty < 65535 ? ty : 65535));
    copy_block_kernel<<<grid, 128, 0, stream>>>(src, lds, dst, ldd, rows, cols);
    CA3DMM_CUDA_TRY(cudaGetLastError());
    ca3dmm_note_launch(1);
    return CA3DMM_OK;
}

// Guard bands of a work buffer: one block, each thread compares its bytes of
// every band with the fill pattern.
__global__ void __launch_bounds__(256)
guard_check_kernel(const unsigned char *__restrict__ base, const ca3dmm_guard_bands_t g,
                   int *status)
{
    for (int b = 0; b < g.n; ++b) {
        const unsigned char *band = base + g.off[b];
        bool bad = false;
        for (int i = threadIdx.x; i < g.bytes; i += blockDim.x)
            bad = bad || band[i] != (unsigned char) g.pattern;
        if (__syncthreads_or(bad) && threadIdx.x == 0 &&
            atomicCAS(status, 0, CA3DMM_DEV_CANARY) == 0)
            status[1] = b;
    }
}

extern "C" int ca3dmm_guard_check_launch(const void *base, const ca3dmm_guard_bands_t *bands,
                                         int *dev_status, cudaStream_t stream)
{
    if (!bands || bands->n <= 0) return CA3DMM_OK;
    if (bands->n > CA3DMM_MAX_CANARIES) return CA3DMM_EINVAL;
    guard_check_kernel<<<1, 256, 0, stream>>>(static_cast<const unsigned char *>(base), *bands,
                                              dev_status);
    CA3DMM_CUDA_TRY(cudaGetLastError());
    ca3dmm_note_launch(1);
    return CA3DMM_OK;
}

extern "C" int ca3dmm_pack_launch(const double *src_base, double *dst_base,
                                  const ca3dmm_pack_desc_t *dev_descs, int ndesc, int total_tiles,
                                  cudaStream_t stream)
{
    if (ndesc <= 0 || total_tiles <= 0) return CA3DMM_OK;
    int grid = ca3dmm_device_sm_count() * 8;
    if (grid > total_tiles) grid = total_tiles;
    pack_kernel<<<grid, 256, 0, stream>>>(src_base, dst_base, dev_descs, ndesc, total_tiles);
    CA3DMM_CUDA_TRY(cudaGetLastError());
    ca3dmm_note_launch(1);
    return CA3DMM_OK;
}

extern "C" int ca3dmm_encode_tmap_2d(void *tmap, int dtype_bytes, const void *base,
                                     unsigned long long dim0, unsigned long long dim1,
                                     unsigned long long stride1_bytes, unsigned box0,
                                     unsigned box1, int swizzle128);

extern "C" int ca3dmm_pack_tma_prepare(ca3dmm_pack_desc_t *descs, int ndesc, const double *src_base,
                                       void *host_tmaps, int *total_tiles)
{
    CUtensorMap *tm = static_cast<CUtensorMap *>(host_tmaps);
    int tiles = 0;
    for (int j = 0; j < ndesc; ++j) {
        ca3dmm_pack_desc_t &d = descs[j];
        memset(&tm[j], 0, sizeof(CUtensorMap));
        d.tile_begin = tiles;
        if (d.rows <= 0 || d.cols <= 0) continue;
        const double *b = src_base + d.src_off;
        if (!d.trans || (d.lds & 1) || (reinterpret_cast<uintptr_t>(b) & 15)) return CA3DMM_EINVAL;
        // source block: cols contiguous doubles per row, rows rows lds apart
        const int rc = ca3dmm_encode_tmap_2d(&tm[j], 8, b, (unsigned long long) d.cols,
                                             (unsigned long long) d.rows,
                                             (unsigned long long) d.lds * 8, TT_BOX, TT_R, 1);
        if (rc) return rc;
        tiles += ((d.rows + TT_R - 1) / TT_R) * ((d.cols + TT_C - 1) / TT_C);
    }
    *total_tiles = tiles;
    return CA3DMM_OK;
}

extern "C" int ca3dmm_pack_tma_launch(const void *dev_tmaps, const ca3dmm_pack_desc_t *dev_descs,
                                      int ndesc, int total_tiles, double *dst_base,
                                      int *dev_status, double timeout_s, cudaStream_t stream)
{
    if (ndesc <= 0 || total_tiles <= 0) return CA3DMM_OK;
    static std::atomic<unsigned long long> attr_done{0};     // one bit per device
    int dev = 0;
    CA3DMM_CUDA_TRY(cudaGetDevice(&dev));
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
    if (!(attr_done.load(std::memory_order_acquire) & bit) || !bit) {
        CA3DMM_CUDA_TRY(cudaFuncSetAttribute(pack_transpose_tma_kernel,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, TT_SMEM));
        attr_done.fetch_or(bit, std::memory_order_release);
    }
    int grid = ca3dmm_device_sm_count();
    if (grid > total_tiles) grid = total_tiles;
    pack_transpose_tma_kernel<<<grid, 256, TT_SMEM, stream>>>(
        static_cast<const CUtensorMap *>(dev_tmaps), dev_descs, ndesc, total_tiles, dst_base,
        dev_status, (unsigned long long) (timeout_s * 1e9));
    CA3DMM_CUDA_TRY(cudaGetLastError());
    ca3dmm_note_launch(1);
    return CA3DMM_OK;
}

extern "C" int ca3dmm_reduce_slabs_launch(const double *slab, long long slab_stride,
                                          long long lds, int nslab, int m, int n, double *out,
                                          long long ldo, cudaStream_t stream)
{
    if (m <= 0 || n <= 0 || nslab <= 0) return CA3DMM_OK;
    int vec = ((reinterpret_cast<uintptr_t>(slab) | reinterpret_cast<uintptr_t>(out)) & 15) == 0 &&
              (lds % 2 == 0) && (ldo % 2 == 0) && (slab_stride % 2 == 0);
    long long work = (vec ? (m + 1LL) / 2 : (long long) m) * n;
    long long blocks = (work + 255) / 256;
    int cap = ca3dmm_device_sm_count() * 8;
    if (blocks > cap) blocks = cap;
    reduce_slabs_kernel<<<(unsigned) blocks, 256, 0, stream>>>(slab, slab_stride, lds, nslab, m, n,
                                                             out, ldo, vec);
    CA3DMM_CUDA_TRY(cudaGetLastError());
    ca3dmm_note_launch(1);
    return CA3DMM_OK;
}

// C(i, j) = C(j, i) for i > j: the strictly lower triangle of an n x n C
// rewritten from the upper one, through 32 x 32 shared-memory tiles (block
// (bi, bj), bi > bj, reads the upper tile (bj, bi) transposed).
__global__ void __launch_bounds__(256)
mirror_upper_kernel(double *__restrict__ C, long long ldc, int n)
{
    __shared__ double t[32][33];
    const int nb = (n + 31) / 32;
    const long long ntile = (long long) nb * (nb + 1) / 2;       // blocks with bi >= bj
    for (long long idx = blockIdx.x; idx < ntile; idx += gridDim.x) {
        // idx -> (bi, bj), bj <= bi, row-major over the lower block triangle
        int bi = (int) ((sqrt(8.0 * (double) idx + 1.0) - 1.0) * 0.5);
        while ((long long) (bi + 1) * (bi + 2) / 2 <= idx) ++bi;
        while ((long long) bi * (bi + 1) / 2 > idx) --bi;
        const int bj = (int) (idx - (long long) bi * (bi + 1) / 2);
        const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
        __syncthreads();                             // t of the previous tile is read
        // read the upper tile: rows 32 bj.., columns 32 bi.. (element (r, c) at r + c ldc)
        for (int y = ty; y < 32; y += 8) {
            const int r = 32 * bj + tx, c = 32 * bi + y;
            t[y][tx] = (r < n && c < n) ? C[r + (long long) c * ldc] : 0.0;
        }
        __syncthreads();
        // write the lower tile: rows 32 bi + tx, columns 32 bj + y, only strictly below the diagonal
        for (int y = ty; y < 32; y += 8) {
            const int r = 32 * bi + tx, c = 32 * bj + y;
            if (r < n && c < n && r > c) C[r + (long long) c * ldc] = t[tx][y];
        }
    }
}

extern "C" int ca3dmm_mirror_upper_launch(double *C, long long ldc, int n, cudaStream_t stream)
{
    if (n <= 1) return CA3DMM_OK;
    const int nb = (n + 31) / 32;
    long long tiles = (long long) nb * (nb + 1) / 2;
    const long long cap = (long long) ca3dmm_device_sm_count() * 8;
    mirror_upper_kernel<<<(unsigned) (tiles < cap ? tiles : cap), 256, 0, stream>>>(C, ldc, n);
    CA3DMM_CUDA_TRY(cudaGetLastError());
    ca3dmm_note_launch(1);
    return CA3DMM_OK;
}

// Diagnostic of the bounded device wait every kernel of the library uses:
// thread 0 waits on an mbarrier that is completed (arrive != 0) or that
// nothing ever completes; the wait returns by itself after limit_ns.
__global__ void wait_check_kernel(int *status, unsigned long long limit_ns, int arrive)
{
    __shared__ uint64_t bar;
    __shared__ volatile int abort_flag;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        abort_flag = 0;
        fence_barrier_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (arrive) mbar_arrive(&bar);
        if (mbar_wait_bounded(&bar, 0, &abort_flag, status, CA3DMM_DEV_TIMEOUT_QUEUE, limit_ns))
            status[1] = 1;
    }
}

extern "C" int ca3dmm_device_wait_check(double timeout_s, int arrive)
{
    if (!(timeout_s >= 0.0) || timeout_s > 60.0) return CA3DMM_EINVAL;
    int *d = nullptr, h[2] = {0, 0};
    CA3DMM_CUDA_TRY(cudaMalloc(&d, 2 * sizeof(int)));
    int rc = CA3DMM_OK;
    if (cudaMemset(d, 0, 2 * sizeof(int)) != cudaSuccess) rc = CA3DMM_ECUDA;
    if (!rc) {
        wait_check_kernel<<<1, 32>>>(d, (unsigned long long) (timeout_s * 1e9), arrive ? 1 : 0);
        ca3dmm_note_launch(1);
        if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess ||
            cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess)
            rc = CA3DMM_ECUDA;
    }
    cudaFree(d);
    if (rc) return rc;
    if (h[0] != 0) return CA3DMM_ETIMEOUT;
    return h[1] ? CA3DMM_OK : CA3DMM_ECUDA;
}
