// SpMM on the tensor cores, for patterns from a few percent nonzeros upwards: the sparse matrix is written
// out densely, 64 columns at a time, in shared memory and multiplied with B, in tensor memory, by tcgen05.mma with
// both operands split into three bf16 parts (mma_split.cuh), six products per fp32 product.
//
// Why: the row-gather kernel pays one L1 wavefront per FMA instruction and ends at 13 to 17 TFLOP/s of stored
// entries, the FMA tile kernel at 45 TFLOP/s of dense arithmetic.  Six bf16 products per fp32 product leave
// 1648 / 6 = 275 TFLOP/s of dense fp32-accurate arithmetic.
//
// A tile is 256 columns of C times up to 128 rows, computed by a PAIR of thread blocks (cta_group::2): the
// columns of C are the tile's M dimension (tensor-memory lanes), the rows of the sparse matrix its N dimension.
// With this orientation a warp's 32 lanes hold 32 neighbouring columns of C and plain 4-byte stores are
// coalesced; and the row count of a tile can be any multiple of 16.  Each block of the pair converts its own
// 128 columns of B and its own half of the rows, and the pair reads both halves of the rows.  (Tiles of 256 rows
// need half the conversions of B per multiply, but the sums then take half of the registers of an SM, and the
// eight operand warps that were left could not hide their latencies: 6000 cycles per 32 columns.)
//
// Sums: the product of the two first parts goes to one accumulator, the five small products to another.  The
// tensor core does not round its sums to nearest, so an accumulator drifts with the number of additions: the
// main one is added to fp32 registers every 64 columns of the sparse matrix, the small one once per tile (its
// drift is relative to sums 2^-8 as large).  A chunk's main product is multiplied first, so that its sums are fetched
// while the five small ones are multiplied: one accumulator of each kind is enough, and the other half of the tensor
// memory holds two stages of B's parts.
//
// B comes by cp.async two chunks ahead, as it is, every warp its own part (also across tiles, so that a tile finds its
// first chunks there), and goes from there split to tensor memory, the first operand of the multiplies.  What bounds the
// kernel are the operand warps: some 360 instructions each per chunk, 63 % of the issue slots (ncu), most of the rest
// their dependences; the tensor pipe needs 1500 of the 2300 cycles of a chunk at 10 % nonzeros.  With B's parts in shared memory
// instead (written once and read by six multiplies, three stages of 72 KiB, 28 KiB left for L1): 2048 x 4096 at 50 %,
// N = 2048 327 -> 297 us, at 10 % 182 -> 180 us, a batch of 256 problems 5540 -> 5060 us, where the entries of the sparse rows
// now find their lines in L1.  Measured and left: B's third part in shared memory and three stages (batch 5460 us; with
// two chunks of raw B 5150 us); rows of B by bulk copies of 512 bytes from one warp (6680 us: it cannot issue them fast
// enough); the entries by cp.async through rings of 128 per row (6560 us: more instructions); two chunks of raw B instead
// of three and the 32 KiB for L1 (5110 us).
//
// Roles of the 28 warps of a block:
//   8 sum warps       add finished accumulators to their registers and write C.
//   16 operand warps  convert 64 rows of B and scatter the matching 64 columns of the sparse rows, eight lanes a
//                     row, into one of two stages; the entries come from registers loaded one chunk ahead.
//   1 issuing warp    (of the even block) issues 24 multiplies a chunk; in the odd block it relays barriers.
//   1 planning warp   lays the next tiles out (problem, place, the rows' entries) for all others.
// (registers are handed out in groups of four warps; the rest of the last group is idle)
//
// Rows whose columns are not strictly ascending, tiles with magnitudes that cannot be split, and sums that are
// not finite are computed again from the CSR arrays with fp32 multiply-adds, so that such input gives what the
// row-gather kernel gives.
#pragma once
#include "mma_split.cuh"
#include "spmm_device.cuh"

namespace dlspm {

constexpr int kMmaChunk = 64;   // columns of the sparse matrix per stage, and per main accumulator
constexpr int kMmaStages = 2;
constexpr int kMmaRawSlots = 3; // chunks of B fetched at once
constexpr int kMmaDepth = 5;    // entries of a row fetched ahead, in eights, of the usual build at most (the deep one: 8)
constexpr int kMmaCols = 128;   // columns of C per block, 256 per pair
constexpr int kMmaRows = 64;    // rows of the sparse matrix per block at most, 128 per pair
constexpr int kMmaMarkWords = 2 * kMmaRows / 32;
constexpr int kMmaSumWarps = 8, kMmaOperandWarps = 16;
constexpr int kMmaThreads = (kMmaSumWarps + kMmaOperandWarps + 4) * 32;
constexpr int kMmaSparsePlane = kMmaChunk * kMmaRows * 2;  // bytes of one part of the sparse operand in a stage
constexpr int kMmaDensePart = kMmaChunk / 2;               // columns of tensor memory of one part of the dense operand
constexpr int kMmaCheckMost = 8192;  // problems of a launch whose columns may be out of order
// Columns of tensor memory: the main accumulator, the one of the small products, two stages of the dense operand.
constexpr uint32_t kMmaSmallColumn = 128, kMmaDenseColumn = 256, kMmaDenseStage = 128;
static_assert(3 * kMmaDensePart <= (int)kMmaDenseStage && kMmaDenseColumn + kMmaStages * kMmaDenseStage <= 512, "tensor memory");
constexpr int kMmaAhead = 4;    // tiles planned ahead
constexpr int kMmaRing = 16;    // tiles whose marks (rows to compute again) can be alive at once
constexpr int kMmaRegsLaunch = 72, kMmaRegsSum = 88, kMmaRegsOperand = 72, kMmaRegsIssue = 40;
static_assert(kMmaThreads * kMmaRegsLaunch <= 65536 &&
                  kMmaSumWarps * 32 * kMmaRegsSum + kMmaOperandWarps * 32 * kMmaRegsOperand + 128 * kMmaRegsIssue <=
                      kMmaThreads * kMmaRegsLaunch,
              "register budgets exceed what the block is launched with");

struct MmaProblem {
    const float *values;
    const int *row_offsets;
    const int *cols;
    const float *B;
    float *C;
    int M, K, N;
    int block_rows;  // rows per tile, a multiple of 16 (half of them per block)
    int row_blocks;  // ceil(M / block_rows)
    int depth;       // entries of a row fetched ahead, in eights: 1 to 8
};

// A tile as the planning warp hands it to the other roles.
struct MmaTile {
    MmaProblem p;                        // (launches over a table)
    int row0, n0;                        // first row and column of this block's part
    int rows;                            // rows per block of the pair
    int chunk0, chunks;                  // its part of K; no chunks: there are no more tiles
    int ring;                            // its marks
    int start[kMmaRows], end[kMmaRows];  // entries of this block's rows
};

struct MmaSmem {
    union {
        unsigned char sparse[kMmaStages][3][kMmaSparsePlane];  // A: rows of 64 columns, 128-byte swizzle
        float part[2 * kMmaRows][kMmaCols];                    // partial sums of a part of K, when the stages are free
        int2 gather[kMmaThreads];                              // pairs of the row-gather loop
    };
    float raw[kMmaRawSlots][kMmaOperandWarps][16 * 32];      // B as it is: 16 rows of 32 columns per warp
    unsigned long long full[kMmaStages], empty[kMmaStages];  // operands written (both blocks) / multiplies done
    unsigned long long sum_full, sum_empty;                  // main accumulator complete / added by all sum warps
    unsigned long long small_full, small_empty;              // the same for the small products, once a tile
    unsigned long long tile_full[kMmaAhead], tile_empty[kMmaAhead];  // tile planned / no longer read
    unsigned long long drain;                                // multiplies still running when a wait ran out
    MmaTile tile[kMmaAhead];
    unsigned again[kMmaRing][kMmaMarkWords];                  // rows of the tile to compute again
    unsigned unsorted[kMmaCheckMost / 32];                   // problems whose columns do not ascend (see mma_looks_sorted)
    uint32_t tmem;
    int abort;
};
constexpr size_t kMmaSmemBytes = sizeof(MmaSmem) + 1024;  // the swizzled planes start at a 1024-byte boundary
static_assert(kMmaSmemBytes <= 232448, "shared memory of a block");

// The tiles of one launch: of a table of problems (tile_start[i] = first tile of problem i), or of one problem.
struct MmaArgs {
    const MmaProblem *problems;
    const long long *tile_start;
    int count;
    int splits;  // parts of K, each a pair of its own; more than one only with one tile per cluster
    long long tiles;
    MmaProblem one;  // used when problems is null
    int before_next;  // the launch behind this one in the stream (with `beside`) may start on SMs as they become free
    int beside;       // this launch needs nothing of the one in front of it and waits for its end at its own end only
    int *error;
};

// A position in the ring of stages and the parity of its barriers' current phase.
struct MmaStage {
    int stage;
    unsigned parity;
    __device__ __forceinline__ void next()
    {
        if (++stage == kMmaStages) {
            stage = 0;
            parity ^= 1u;
        }
    }
};

// ---- planning warp ------------------------------------------------------------------------------------

// Where the walk over the tiles of a cluster is.
struct MmaPlan {
    long long tile;
    int prob;
    const MmaProblem *p;
    int cb, rb;  // 256 columns, block_rows rows
};

template <bool TABLE>
__device__ __forceinline__ bool mma_plan_load(MmaPlan &t, const MmaArgs &a)
{
    if (t.tile >= a.tiles) return false;
    long long first = 0;
    if constexpr (TABLE) {
        int lo = t.prob, hi = a.count - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(a.tile_start + mid) <= t.tile) lo = mid;
            else hi = mid - 1;
        }
        t.prob = lo;
        t.p = a.problems + lo;
        first = __ldg(a.tile_start + lo);
    } else {
        t.p = &a.one;
    }
    const int i = (int)(t.tile - first);
    t.cb = i / t.p->row_blocks;
    t.rb = i - t.cb * t.p->row_blocks;
    return true;
}

// The same, past tiles of problems that were computed at the start of the kernel.
template <bool TABLE, bool CHECK>
__device__ __forceinline__ bool mma_plan_next(MmaPlan &t, const MmaArgs &a, const MmaSmem &sm)
{
    while (mma_plan_load<TABLE>(t, a)) {
        if (!(TABLE && CHECK) || !((sm.unsorted[t.prob >> 5] >> (t.prob & 31)) & 1u)) return true;
        t.tile += gridDim.x / (2u * (unsigned)a.splits);
    }
    return false;
}

// Lays tile n of this cluster out; false behind the last one.
template <bool TABLE, bool CHECK>
__device__ __forceinline__ bool mma_plan_tile(MmaSmem &sm, const MmaArgs &a, unsigned rank, int lane, MmaPlan &t, unsigned n)
{
    const bool more = mma_plan_next<TABLE, CHECK>(t, a, sm);
    MmaTile &out = sm.tile[n % kMmaAhead];
    if (more) {
        const int rows = t.p->block_rows >> 1, row0 = t.rb * t.p->block_rows;
        int start[kMmaRows / 32], end[kMmaRows / 32];
#pragma unroll
        for (int i = 0; i < kMmaRows / 32; i++) {  // (all of them in flight)
            const int r = lane + 32 * i, row = row0 + (int)(rank & 1u) * rows + r;
            start[i] = end[i] = 0;
            if (r < rows && row < t.p->M) {
                start[i] = __ldg(t.p->row_offsets + row);
                end[i] = __ldg(t.p->row_offsets + row + 1);
            }
        }
        if constexpr (TABLE) {
            static_assert(sizeof(MmaProblem) == 64, "copied by sixteen lanes");
            if (lane < 16) reinterpret_cast<int *>(&out.p)[lane] = __ldg(reinterpret_cast<const int *>(t.p) + lane);
        }
        if (lane == 0) {
            const int all = (t.p->K + kMmaChunk - 1) / kMmaChunk, part = (int)(rank >> 1), shift = __ffs(a.splits) - 1;  // splits: 1, 2 or 4
            out.rows = rows;
            out.row0 = row0;
            out.n0 = t.cb * 2 * kMmaCols + (int)(rank & 1u) * kMmaCols;
            out.chunk0 = (all * part) >> shift;
            out.chunks = ((all * (part + 1)) >> shift) - out.chunk0;
            out.ring = (int)(n % kMmaRing);
        }
#pragma unroll
        for (int i = 0; i < kMmaRows / 32; i++) {
            out.start[lane + 32 * i] = start[i];
            out.end[lane + 32 * i] = end[i];
        }
        t.tile += gridDim.x / (2u * (unsigned)a.splits);
    } else if (lane == 0) {
        out.chunks = 0;
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.tile_full[n % kMmaAhead]);
    return more;
}

// Tiles n, n + 1, .. up to kMmaAhead ahead of the other roles, so that none of them meets the chain of dependent loads
// (which problem, its sizes and addresses, the rows' offsets) between two tiles: with every role looking its tiles up by
// itself a tile cost 2 to 3 us more (37 problems of 2048 x 512 at 10 %, N = 3136, eight chunks a tile: 2.06 -> 1.65 us per
// chunk of 64 columns; of 1024 x 4096, N = 1024, 64 chunks a tile: 1.75 -> 1.62; a batch of 256 problems 6040 -> 5640 us).
template <bool TABLE, bool CHECK>
__device__ __forceinline__ bool mma_plan(MmaSmem &sm, const MmaArgs &a, unsigned rank, int lane, MmaPlan &t, unsigned n)
{
    for (;; n++) {
        if (!mbar_wait_suspended(&sm.tile_empty[n % kMmaAhead], ((n / kMmaAhead) & 1u) ^ 1u, &sm.abort)) return false;
        if (!mma_plan_tile<TABLE, CHECK>(sm, a, rank, lane, t, n)) return true;
    }
}

// A role's walk over the planned tiles.
struct MmaWalk {
    unsigned n = 0;
    // Waits for the tile; false if a wait ran out.
    __device__ __forceinline__ bool wait(MmaSmem &sm) const
    {
        return mbar_wait_suspended(&sm.tile_full[n % kMmaAhead], (n / kMmaAhead) & 1u, &sm.abort);
    }
    __device__ __forceinline__ const MmaTile &tile(const MmaSmem &sm) const { return sm.tile[n % kMmaAhead]; }
    // By one thread per warp (or relay), when the tile is no longer read.
    __device__ __forceinline__ void done(MmaSmem &sm) { mbar_arrive(&sm.tile_empty[n % kMmaAhead]); }
};
// The problem of a tile: of a lone launch among the kernel's arguments, where its fields cost no registers.
template <bool TABLE>
__device__ __forceinline__ const MmaProblem &mma_problem_of(const MmaTile &t, const MmaArgs &a)
{
    if constexpr (TABLE) return t.p;
    else return a.one;
}

// First entries at or behind column `col` of the rows of a warp, eight lanes a row, 32 probes a round: two or three
// rounds of dependent loads for a row, where halving took twelve (with the planning, 1024 x 4096 at 10 %, N = 1024 in two
// parts: 59.2 -> 57.2 us).
__device__ __forceinline__ int mma_lower_bound(const int *__restrict__ cols, int lo, int hi, int col, int l8)
{
    while (__any_sync(0xffffffffu, lo < hi)) {
        const int step = max(1, (hi - lo + 31) / 32);
        int below = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int at = lo + (4 * l8 + i) * step;
            if (at < hi && __ldg(cols + at) < col) below++;
        }
#pragma unroll
        for (int d = 1; d < 8; d <<= 1) below += __shfl_xor_sync(0xffffffffu, below, d);
        if (lo < hi) {
            const int l = lo;
            if (below > 0) lo = l + (below - 1) * step + 1;
            hi = min(hi, l + below * step);
        }
    }
    return lo;
}

// ---- operand warps ------------------------------------------------------------------------------------

// The fetches of an operand warp's part of B, rows 16 * (warp / 4) .. + 15 of a chunk and columns 32 * (warp % 4) .. + 31 of
// this block's, two chunks ahead of the conversion and across tiles.  Rows and columns past the end of B are others of
// its own: no entry refers to such a row, and such a column is not stored.
struct MmaFetch {
    unsigned n;        // tile
    int left;          // its chunks to come; < 0: behind the last tile
    int rows;          // rows of B from this warp's first one of the next chunk on
    const char *next;  // this lane's first element of the next chunk
    unsigned row;      // bytes from row to row
};

__device__ __forceinline__ void copy_async16(uint32_t dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async4(uint32_t dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void copy_async_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory");
}

// The tile's place in B; false if a wait ran out.
template <bool TABLE, bool WIDE>
__device__ __forceinline__ bool mma_fetch_tile(MmaFetch &f, MmaSmem &sm, const MmaArgs &a, int warp, int lane)
{
    if (!mbar_wait_suspended(&sm.tile_full[f.n % kMmaAhead], (f.n / kMmaAhead) & 1u, &sm.abort)) return false;
    const MmaTile &t = sm.tile[f.n % kMmaAhead];
    const MmaProblem &p = mma_problem_of<TABLE>(t, a);
    f.left = t.chunks == 0 ? -1 : t.chunks;
    if (f.left < 0) return true;
    int n = t.n0 + 32 * (warp & 3) + (WIDE ? 4 * (lane & 7) : lane);
    // Columns past the end: others instead, by steps of 32, so that the lanes of a request differ.  (Copies of one word to 32
    // places are done one by one: all on the last column, 3000 x 1500 at 50 %, N = 770 took 227 us.)
    if (n >= p.N) n = max(n - ((n - p.N) / 32 + 1) * 32, 0);
    n = min(n, p.N - (WIDE ? 4 : 1));
    const int k = t.chunk0 * kMmaChunk + 16 * (warp >> 2);
    f.rows = p.K - k;
    f.row = 4u * (unsigned)p.N;
    f.next = reinterpret_cast<const char *>(p.B) + 4 * ((size_t)(k + (WIDE ? lane >> 3 : 0)) * (size_t)p.N + (size_t)n);
    return true;
}

// Requests the next chunk into `dst`, the warp's part of a slot.
template <bool TABLE, bool WIDE>
__device__ __forceinline__ bool mma_fetch(MmaFetch &f, MmaSmem &sm, const MmaArgs &a, int warp, int lane, uint32_t dst)
{
    if (f.left == 0) {
        f.n++;
        if (!mma_fetch_tile<TABLE, WIDE>(f, sm, a, warp, lane)) return false;
    }
    if (f.left > 0) {
        f.left--;
        constexpr int kStep = WIDE ? 4 : 1;  // rows a request of the warp covers
        dst += (WIDE ? 16u : 4u) * (unsigned)lane;
        const char *src = f.next;
        if (f.rows >= 16) {
#pragma unroll
            for (int i = 0; i < 16 / kStep; i++) {
                if constexpr (WIDE) copy_async16(dst + 128 * kStep * i, src);
                else copy_async4(dst + 128 * i, src);
                src += kStep * f.row;
            }
        } else {  // (the last chunk of a problem)
            const int first = WIDE ? lane >> 3 : 0;
            for (int i = 0; i < 16; i += kStep) {
                const char *at = src + (long long)(min(first + i, f.rows - 1) - first) * (long long)f.row;
                if constexpr (WIDE) copy_async16(dst + 128 * i, at);
                else copy_async4(dst + 128 * i, at);
            }
        }
        f.next += 64ull * f.row;
        f.rows -= 64;
    }
    copy_async_commit();
    return true;
}

// Writes eight rows split to tensor memory: a lane is a column of B, a 32-bit word two neighbouring rows.
__device__ __forceinline__ void mma_store_dense(uint32_t dst, const float *raw, unsigned &least)
{
    float d[8];
#pragma unroll
    for (int i = 0; i < 8; i++) d[i] = raw[32 * i];
    uint32_t x1[4], x2[4], x3[4];
    float small = 1.f;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        small = min3_magnitude(small, d[2 * i], d[2 * i + 1]);
        split_pair(d[2 * i], d[2 * i + 1], x1[i], x2[i], x3[i]);
    }
    __syncwarp();
    tmem_store4(dst, x1);
    tmem_store4(dst + kMmaDensePart, x2);
    tmem_store4(dst + 2 * kMmaDensePart, x3);
    // a zero, or a number that cannot be split (asked by the whole warp: the wait for the stores is for a converged one)
    if (__any_sync(0xffffffffu, small < kSplitSmall)) {
#pragma unroll
        for (int i = 0; i < 8; i++) least = split_magnitude(d[i], least);
    }
}

// Entries q, q + 8, .. of a row; slots past its end hold a column that no chunk contains.
template <int DEPTH>
__device__ __forceinline__ void mma_load_pairs(int (&c)[DEPTH], float (&v)[DEPTH], int q, int end, const MmaProblem &p)
{
    const char *cols = reinterpret_cast<const char *>(p.cols), *values = reinterpret_cast<const char *>(p.values);
    const unsigned at = 4u * (unsigned)q;
#pragma unroll
    for (int h = 0; h < DEPTH; h++) {
        c[h] = 0x7fffffff;
        if (q + 8 * h < end) {
            c[h] = __ldg(reinterpret_cast<const int *>(cols + (at + 32u * h)));
            v[h] = __ldg(reinterpret_cast<const float *>(values + (at + 32u * h)));
        }
    }
}

// One entry of the sparse matrix into a stage; `row` is the address of its row of the first part.
__device__ __forceinline__ void mma_store_entry(uint32_t row, int col, float v, int swizzle, bool live)
{
    uint32_t p1, p2, p3;
    split_one(v, p1, p2, p3);
    const uint32_t e = row + ((col * 2) ^ swizzle);
    if (live) {
        store_shared_half(e, p1);
        store_shared_half(e + kMmaSparsePlane, p2);
        store_shared_half(e + 2 * kMmaSparsePlane, p3);
    }
}

__device__ __forceinline__ void mma_mark_again(MmaSmem &sm, int ring, int bit, unsigned rank)
{
    mark_in_pair(&sm.again[ring][bit >> 5], 1u << (bit & 31), rank);
}

// One tile: every lane group of eight lanes owns one row of it, 4 * warp + group, and walks it once.  DEPTH: entries
// of a row fetched ahead, in eights.  CHECK: columns may be out of order (a prepared batch looked at them when it was
// made).
template <int DEPTH, bool TABLE, bool WIDE, bool CHECK>
__device__ __forceinline__ bool mma_operand_tile(MmaSmem &sm, const MmaArgs &a, const MmaTile &t, unsigned rank, int warp, int lane, MmaStage &st,
                                                 MmaFetch &f, unsigned &slot)
{
    volatile int *abort = &sm.abort;
    const MmaProblem &p = mma_problem_of<TABLE>(t, a);
    const int l8 = lane & 7, group = lane & 24, own = warp * 4 + (lane >> 3);
    const int swizzle = (own & 7) << 4;
    const int chunks = t.chunks;
    const bool row_warp = warp * 4 < t.rows;  // this warp has rows in the tile
    int cursor = t.start[own], end = t.end[own];
    if (a.splits > 1) {
        const int part = (int)(rank >> 1), first = cursor, stop = end;
        if (part > 0) cursor = mma_lower_bound(p.cols, first, stop, t.chunk0 * kMmaChunk, l8);
        if (part + 1 < a.splits) end = mma_lower_bound(p.cols, first, stop, (t.chunk0 + t.chunks) * kMmaChunk, l8);
    }
    int k0 = t.chunk0 * kMmaChunk;
    const uint32_t dense_at = sm.tmem + ((uint32_t)(warp & 3) << 21) + kMmaDenseColumn + 8u * (unsigned)(warp >> 2);
    const uint32_t sparse_at = smem_u32(&sm.sparse[0][0][0]) + own * 128;
    unsigned least = 0xffffffffu;
    bool bad = false, ok = true;  // bad: the lane group's row has columns out of order
    // One chunk: its entries are in (c, v), the next chunk's are fetched into (cn, vn).
    auto step = [&](int (&c)[DEPTH], float (&v)[DEPTH], int (&cn)[DEPTH], float (&vn)[DEPTH]) {
        copy_async_wait<1>();
        __syncwarp();  // this chunk has landed, and the one before it has been read
        const float *raw = sm.raw[slot][warp] + lane;
        const unsigned behind = slot == 0u ? kMmaRawSlots - 1u : slot - 1u;
        ok = mma_fetch<TABLE, WIDE>(f, sm, a, warp, lane, smem_u32(sm.raw[behind][warp])) &&
             mbar_wait_suspended(&sm.empty[st.stage], st.parity ^ 1u, abort);  // passes at once in the first round
        slot = slot == kMmaRawSlots - 1u ? 0u : slot + 1u;
        if (!ok) return;
        tmem_fence_after();
        const uint32_t row = sparse_at + st.stage * (3 * kMmaSparsePlane);
        const uint32_t dst = dense_at + st.stage * kMmaDenseStage;
        int turns = 0;  // eights of entries at hand of which some row uses one
        if (row_warp) {
            // this warp's four rows: zeros in all three parts
            const uint32_t z = row + l8 * 16;
            store_shared_zero(z);
            store_shared_zero(z + kMmaSparsePlane);
            store_shared_zero(z + 2 * kMmaSparsePlane);
            __syncwarp();
            // how many of the entries at hand belong to this chunk (they are the first of them: columns ascend)
            int used = 0;
#pragma unroll
            for (int h = 0; h < DEPTH; h++) {
                const unsigned m = __ballot_sync(0xffffffffu, (unsigned)(c[h] - k0) < (unsigned)kMmaChunk);
                used += __popc((m >> group) & 0xffu);
                if (DEPTH > 5 && m) turns = h + 1;
            }
            cursor += used;
            bool more = used == 8 * DEPTH;
            while (__any_sync(0xffffffffu, more)) {  // more entries than were fetched ahead: eight at a time
                const int q = cursor + l8;
                bool take = false;
                if (more && q < end) {
                    const int col = __ldg(p.cols + q), before = CHECK ? __ldg(p.cols + q - 1) : -1;
                    const float x = __ldg(p.values + q);
                    take = (unsigned)(col - k0) < (unsigned)kMmaChunk;
                    if (take) {
                        if (CHECK && col <= before) bad = true;
                        least = split_magnitude(x, least);
                        mma_store_entry(row, col - k0, x, swizzle, true);
                    }
                }
                const int got = __popc((__ballot_sync(0xffffffffu, take) >> group) & 0xffu);
                cursor += got;
                more = got == 8;
            }
            if constexpr (DEPTH <= 2) mma_load_pairs(cn, vn, cursor + l8, end, p);
        }
        mma_store_dense(dst, raw, least);
        if (row_warp) {
            int last = -1;  // column in front of the first entry at hand (entries of earlier chunks are in order)
#pragma unroll
            for (int h = 0; h < DEPTH; h++) {
                if (DEPTH > 5 && h >= turns) break;  // the whole warp
                const int col = c[h] - k0;
                const bool live = (unsigned)col < (unsigned)kMmaChunk;
                if constexpr (CHECK) {
                    int before = __shfl_up_sync(0xffffffffu, col, 1, 8);
                    if (l8 == 0) before = last;
                    if (h + 1 < DEPTH) last = __shfl_sync(0xffffffffu, col, 7, 8);
                    bad = bad || (live && col <= before);
                }
                if (live) least = split_magnitude(v[h], least);
                mma_store_entry(row, col, v[h], swizzle, live);
            }
            if constexpr (DEPTH > 2) mma_load_pairs(c, v, cursor + l8, end, p);
        }
        mma_store_dense(dst + 4, raw + 8 * 32, least);
        k0 += kMmaChunk;
    };
    // Hands a stage over; `marks`: the tile's last one.
    auto hand_over = [&](bool marks) {
        if (marks) {
            if (CHECK && cursor != end) bad = true;  // entries out of order were never reached
            const bool all = __any_sync(0xffffffffu, least < kSplitLeast);
            if (__any_sync(0xffffffffu, bad) || all) {
                if (bad && own < t.rows) mma_mark_again(sm, t.ring, (int)(rank & 1u) * t.rows + own, rank);
                if (all)
                    for (int r = lane; r < 2 * t.rows; r += 32) mma_mark_again(sm, t.ring, r, rank);
                __syncwarp();
            }
        }
        tmem_store_wait();
        tmem_fence_before();
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.full[st.stage]);
        st.next();
    };
    int c0[DEPTH];
    float v0[DEPTH];
    mma_load_pairs(c0, v0, cursor + l8, end, p);
    if constexpr (DEPTH <= 2) {
        // two chunks a turn with the register sets exchanged: copying one to the other would wait for its loads
        int c1[DEPTH];
        float v1[DEPTH];
        for (int i = 0; i < chunks; i += 2) {
            step(c0, v0, c1, v1);
            if (!ok) return false;
            hand_over(i + 1 == chunks);
            if (i + 1 < chunks) {
                step(c1, v1, c0, v0);
                if (!ok) return false;
                hand_over(i + 2 == chunks);
            }
        }
    } else {
        // (no registers for a second set; the entries of a dense chunk are fetched behind the last one's)
        for (int i = 0; i < chunks; i++) {
            step(c0, v0, c0, v0);
            if (!ok) return false;
            hand_over(i + 1 == chunks);
        }
    }
    return true;
}

template <bool TABLE, bool WIDE, bool DEEP, bool CHECK>
__device__ __forceinline__ bool mma_operands(MmaSmem &sm, const MmaArgs &a, unsigned rank, int warp, int lane)
{
    MmaStage st{0, 0u};
    MmaFetch f;
    f.n = 0u;
    unsigned slot = 0u;
    bool ok = mma_fetch_tile<TABLE, WIDE>(f, sm, a, warp, lane);
#pragma unroll
    for (int i = 0; i + 1 < kMmaRawSlots; i++) ok = ok && mma_fetch<TABLE, WIDE>(f, sm, a, warp, lane, smem_u32(sm.raw[i][warp]));
    for (MmaWalk walk; ok; walk.n++) {
        ok = walk.wait(sm);
        if (!ok) break;
        const MmaTile &t = walk.tile(sm);
        if (t.chunks == 0) break;
        if constexpr (DEEP) {
            ok = mma_operand_tile<8, TABLE, WIDE, CHECK>(sm, a, t, rank, warp, lane, st, f, slot);
        } else {
            const int depth = mma_problem_of<TABLE>(t, a).depth;
            if (depth == 1) ok = mma_operand_tile<1, TABLE, WIDE, CHECK>(sm, a, t, rank, warp, lane, st, f, slot);
            else if (depth == 2) ok = mma_operand_tile<2, TABLE, WIDE, CHECK>(sm, a, t, rank, warp, lane, st, f, slot);
            else ok = mma_operand_tile<5, TABLE, WIDE, CHECK>(sm, a, t, rank, warp, lane, st, f, slot);
        }
        __syncwarp();
        if (ok && lane == 0) walk.done(sm);
    }
    copy_async_wait<0>();
    return ok;
}

// ---- issuing warp (of the even block) ----------------------------------------------------------

// The whole warp walks the chunks, one lane issues (the instructions take their operands from uniform registers,
// which the compiler can only use where control flow is uniform).
__device__ __forceinline__ bool mma_issue(MmaSmem &sm, unsigned rank, bool issuer, int lane)
{
    volatile int *abort = &sm.abort;
    const unsigned pair_mask = 3u << rank;
    const uint32_t tmem = sm.tmem;
    // parts (of B, of A) of the five small products
    const int part_b[5] = {2, 1, 1, 0, 0}, part_a[5] = {0, 1, 0, 2, 1};
    const uint64_t sparse0 = mma_descriptor(smem_u32(&sm.sparse[0][0][0]), 0, 1024, kSwizzle128);
    constexpr uint64_t kSparse = kMmaSparsePlane >> 4;
    const uint32_t main = tmem, small = tmem + kMmaSmallColumn;
    unsigned g = 0;  // chunks so far
    for (MmaWalk walk;; walk.n++) {
        if (!walk.wait(sm)) return false;
        const int chunks = walk.tile(sm).chunks, rows = walk.tile(sm).rows;
        __syncwarp();
        if (lane == 0) walk.done(sm);
        if (chunks == 0) return true;
        const uint32_t instruction = mma_instruction(256, 2 * rows, false, false);
        for (int c = 0; c < chunks; c++, g++) {
            const int s = (int)(g % kMmaStages);
            if (!mbar_wait_suspended(&sm.full[s], (g / kMmaStages) & 1u, abort)) return false;
            if (!mbar_wait_suspended(&sm.sum_empty, (g & 1u) ^ 1u, abort)) return false;  // passes at once the first time
            tmem_fence_after();
            const uint32_t dense = tmem + kMmaDenseColumn + s * kMmaDenseStage;
            const uint64_t sparse = sparse0 + s * (3 * kSparse);
            if (issuer) {
#pragma unroll
                for (int ks = 0; ks < kMmaChunk / 16; ks++)
                    mma_bf16_tmem(main, dense + ks * 8, sparse + ks * (32 >> 4), instruction, ks > 0);
                mma_commit<true>(&sm.sum_full, pair_mask);
            }
            __syncwarp();
            if (c == 0) {  // the small sums of the tile before have been read
                if (!mbar_wait_suspended(&sm.small_empty, (walk.n & 1u) ^ 1u, abort)) return false;
                tmem_fence_after();
            }
            if (issuer) {
#pragma unroll
                for (int ks = 0; ks < kMmaChunk / 16; ks++)
#pragma unroll
                    for (int j = 0; j < 5; j++)
                        mma_bf16_tmem(small, dense + part_b[j] * kMmaDensePart + ks * 8, sparse + part_a[j] * kSparse + ks * (32 >> 4),
                                      instruction, c + j + ks > 0);
                mma_commit<true>(&sm.empty[s], pair_mask);
                if (c + 1 == chunks) mma_commit<true>(&sm.small_full, pair_mask);
            }
            __syncwarp();
        }
    }
}

// ---- relay (odd block) ------------------------------------------------------------------------------------

// Passes the odd block's barriers on to the even block's, one arrival per phase: a remote arrival orders all
// memory accesses of its thread first, which would hold up a warp with loads in flight.  (One thread.)
__device__ __forceinline__ bool mma_relay(MmaSmem &sm, unsigned rank, bool sums)
{
    volatile int *abort = &sm.abort;
    const unsigned slots = sums ? 1u : (unsigned)kMmaStages;
    unsigned long long *own = sums ? &sm.sum_empty : sm.full;
    const uint32_t other = cluster_map(smem_u32(own), rank ^ 1u), other_small = cluster_map(smem_u32(&sm.small_empty), rank ^ 1u);
    unsigned g = 0;
    for (MmaWalk walk;; walk.n++) {
        if (!walk.wait(sm)) return false;
        const int chunks = walk.tile(sm).chunks;
        walk.done(sm);
        if (chunks == 0) return true;
        for (int c = 0; c < chunks; c++, g++) {
            if (!mbar_wait_suspended(&own[g % slots], (g / slots) & 1u, abort)) return false;
            tmem_fence_after();
            tmem_fence_before();
            mbar_arrive_cluster(other + (g % slots) * 8u);
        }
        if (sums) {
            if (!mbar_wait_suspended(&sm.small_empty, walk.n & 1u, abort)) return false;
            tmem_fence_after();
            tmem_fence_before();
            mbar_arrive_cluster(other_small);
        }
    }
}

// ---- sum warps --------------------------------------------------------------------------------------------

__device__ __forceinline__ void sum_warps_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kMmaSumWarps * 32) : "memory"); }

// Row `row` of C, this block's 128 columns from n0, by one warp from the CSR arrays.
__device__ __forceinline__ void mma_row_again(const MmaProblem &p, int row, int n0, int lane)
{
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int q = __ldg(p.row_offsets + row), end = __ldg(p.row_offsets + row + 1); q < end; q++) {
        const float v = __ldg(p.values + q);
        const float *b = p.B + (size_t)__ldg(p.cols + q) * (size_t)p.N + n0 + lane;
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (n0 + lane + 32 * i < p.N) acc[i] = fmaf(v, __ldg(b + 32 * i), acc[i]);
    }
    float *c = p.C + (size_t)row * (size_t)p.N + n0 + lane;
#pragma unroll
    for (int i = 0; i < 4; i++)
        if (n0 + lane + 32 * i < p.N) c[32 * i] = acc[i];
}

// Marks the columns of the accumulators (rows of the sparse matrix) in which some lane holds a sum that is not
// finite.  `first` is the row of acc[0].
template <int COUNT>
__device__ __forceinline__ void mma_mark_not_finite(MmaSmem &sm, int ring, const float (&acc)[COUNT], int first, int lane)
{
    float probe[2] = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < COUNT; j++) probe[j & 1] = fmaf(acc[j], 0.f, probe[j & 1]);
    if (!__any_sync(0xffffffffu, probe[0] + probe[1] != 0.f)) return;  // NaN compares unequal
#pragma unroll
    for (int j = 0; j < COUNT; j++)
        if (__any_sync(0xffffffffu, fmaf(acc[j], 0.f, 0.f) != 0.f) && lane == 0)
            atomicOr(&sm.again[ring][(first + j) >> 5], 1u << ((first + j) & 31));
}

// Warp w: tensor-memory lanes 32 * (w % 4) .. + 31 (columns of C), accumulator columns 64 * (w / 4) .. + 63
// (rows of the sparse matrix).
template <bool TABLE>
__device__ __forceinline__ bool mma_sums(MmaSmem &sm, const MmaArgs &a, unsigned rank, int warp, int lane)
{
    volatile int *abort = &sm.abort;
    const int half = (warp >> 2) * kMmaRows, quarter = warp & 3;
    const uint32_t tmem = sm.tmem + ((uint32_t)quarter << 21) + (uint32_t)half;
    unsigned q = 0;
    for (MmaWalk walk;; walk.n++) {
        if (!walk.wait(sm)) return false;
        const MmaTile &t = walk.tile(sm);
        const int chunks = t.chunks;
        if (chunks == 0) return true;
        const int tile_rows = 2 * t.rows;
        float acc[kMmaRows];
#pragma unroll
        for (int j = 0; j < kMmaRows; j++) acc[j] = 0.f;
        for (int i = 0; i < chunks; i++, q++) {
            if (!mbar_wait_suspended(&sm.sum_full, q & 1u, abort)) return false;
            tmem_fence_after();
            tmem_add(acc, tmem, tile_rows - half);
            tmem_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.sum_empty);
        }
        if (!mbar_wait_suspended(&sm.small_full, walk.n & 1u, abort)) return false;
        tmem_fence_after();
        tmem_add(acc, tmem + kMmaSmallColumn, tile_rows - half);
        tmem_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.small_empty);
        if (a.splits > 1) {
            // partial sums to shared memory (the stages are free: this was the last tile); the blocks of the
            // cluster that hold the same columns add them up behind a cluster barrier, in mma_combine
#pragma unroll
            for (int j = 0; j < kMmaRows; j++) sm.part[half + j][32 * quarter + lane] = acc[j];
            return true;
        }
        const int ring = t.ring;
        mma_mark_not_finite(sm, ring, acc, half, lane);
        const MmaProblem &p = mma_problem_of<TABLE>(t, a);
        const int n = t.n0 + 32 * quarter + lane;
        if (n < p.N) {
            const int N = p.N, rows = min(tile_rows, p.M - t.row0) - half;
            float *c = p.C + (size_t)(t.row0 + half) * (size_t)N + n;
#pragma unroll
            for (int j = 0; j < kMmaRows; j++)
                if (j < rows) __stcs(c + (size_t)j * (size_t)N, acc[j]);
        }
        sum_warps_barrier();
        unsigned any = 0;
        for (int w = 0; w < kMmaMarkWords; w++) any |= *(volatile unsigned *)&sm.again[ring][w];
        if (any) {
            for (int j = warp; j < tile_rows; j += kMmaSumWarps)
                if (((*(volatile unsigned *)&sm.again[ring][j >> 5] >> (j & 31)) & 1u) && t.row0 + j < p.M)
                    mma_row_again(p, t.row0 + j, t.n0, lane);
            sum_warps_barrier();
            if (warp == 0 && lane < kMmaMarkWords) sm.again[ring][lane] = 0u;
        }
        __syncwarp();
        if (lane == 0) walk.done(sm);
    }
}

// splits > 1: adds the partial sums of the tile over the parts of K, in order.  Block part p takes the rows of
// the tile's p-th share.
template <bool TABLE>
__device__ __forceinline__ void mma_combine(MmaSmem &sm, const MmaArgs &a, unsigned rank, int warp, int lane)
{
    const MmaTile &t = sm.tile[0];  // the only one
    const MmaProblem &p = mma_problem_of<TABLE>(t, a);
    const int tile_rows = 2 * t.rows, part = (int)(rank >> 1);
    const int per = (tile_rows + a.splits - 1) / a.splits;
    const int first = part * per, last = min(min(first + per, tile_rows), p.M - t.row0);
    const uint32_t sums = smem_u32(&sm.part[0][0]);
    uint32_t again = 0;  // lane w < 4: word w of the marks of all parts
    if (lane < kMmaMarkWords)
        for (int s = 0; s < a.splits; s++)
            again |= cluster_load_u32(cluster_map(smem_u32(&sm.again[0][lane]), (unsigned)(2 * s) | (rank & 1u)));
    for (int j = first + warp; j < last; j += kMmaSumWarps) {
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        for (int s = 0; s < a.splits; s++) {
            const uint32_t from = cluster_map(sums + (uint32_t)(j * kMmaCols + lane) * 4u, (unsigned)(2 * s) | (rank & 1u));
#pragma unroll
            for (int i = 0; i < 4; i++) v[i] += cluster_load(from + 128u * i);
        }
        float probe = 0.f;
#pragma unroll
        for (int i = 0; i < 4; i++) probe = fmaf(v[i], 0.f, probe);
        const unsigned word = __shfl_sync(0xffffffffu, again, j >> 5);
        if (__any_sync(0xffffffffu, probe != 0.f) || ((word >> (j & 31)) & 1u)) {
            mma_row_again(p, t.row0 + j, t.n0, lane);
        } else {
            float *c = p.C + (size_t)(t.row0 + j) * (size_t)p.N + t.n0 + lane;
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (t.n0 + lane + 32 * i < p.N) c[32 * i] = v[i];
        }
    }
}

// ---- columns out of order ---------------------------------------------------------------------------------------

// Looks at eight entries each of 32 rows.  Rows out of order that this does not find are computed again one by one; a
// pattern whose rows are out of order as a rule (as some formats leave them) would take ten times as long that way as
// with the row-gather loop, which the kernel then runs instead.
__device__ __forceinline__ bool mma_looks_sorted(const MmaProblem &p, int lane)
{
    const int row = (int)((long long)p.M * lane / 32);
    const int start = __ldg(p.row_offsets + row), end = __ldg(p.row_offsets + row + 1);
    const int from = start + (end - start) / 2;
    int c[8];
#pragma unroll
    for (int i = 0; i < 8; i++) c[i] = from + i < end ? __ldg(p.cols + from + i) : 0x7fffffff;
    bool ok = true;
#pragma unroll
    for (int i = 1; i < 8; i++) ok = ok && (c[i] > c[i - 1] || from + i >= end);
    return __all_sync(0xffffffffu, ok);
}

// A whole problem with the row-gather loop, by all warps of the launch.
template <int VEC>
__device__ __forceinline__ void mma_gather(const MmaProblem &p, int2 *stage, int warp, int lane)
{
    constexpr int kCols = 32 * VEC;
    const long long items = (long long)p.M * ((p.N + kCols - 1) / kCols);
    for (long long i = (long long)blockIdx.x * (kMmaThreads / 32) + warp; i < items; i += (long long)gridDim.x * (kMmaThreads / 32)) {
        const int slab = (int)(i / p.M), row = (int)(i - (long long)slab * p.M);
        spmm_warp_row_slab<VEC, 1, false, 4>(p.values, p.cols, __ldg(p.row_offsets + row), __ldg(p.row_offsets + row + 1), p.B,
                                             p.C + (size_t)row * (size_t)p.N, p.N, slab * kCols, lane, stage);
    }
}

// Grid: clusters of 2 * splits blocks; cluster i takes the tiles i, i + clusters, ...  error[0] is set to 1 if a
// bounded wait ran out.
// TABLE: the tiles of a table of problems; otherwise of the one problem among the arguments (whose fields then cost
// no registers).  WIDE: rows of B are 16-byte aligned.  DEEP: the build for problems with more than 40 entries of a
// row ahead (in one build with the others its registers cost those 10 to 20 %).  CHECK: columns may be out of order.
template <bool TABLE, bool WIDE, bool DEEP, bool CHECK>
__global__ void __launch_bounds__(kMmaThreads, 1) spmm_mma_kernel(const __grid_constant__ MmaArgs a)
{
    extern __shared__ unsigned char smem_raw[];
    MmaSmem &sm = *reinterpret_cast<MmaSmem *>(smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned rank = cluster_rank();
    constexpr int kIssueWarp = kMmaSumWarps + kMmaOperandWarps, kPlanWarp = kIssueWarp + 2;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kMmaStages; s++) {
            mbar_init(&sm.full[s], kMmaOperandWarps + (rank & 1u ? 0u : 1u));  // even block: plus the odd one's relay
            mbar_init(&sm.empty[s], 1);
        }
        mbar_init(&sm.sum_full, 1);
        mbar_init(&sm.sum_empty, kMmaSumWarps + (rank & 1u ? 0u : 1u));
        mbar_init(&sm.small_full, 1);
        mbar_init(&sm.small_empty, kMmaSumWarps + (rank & 1u ? 0u : 1u));
        for (int n = 0; n < kMmaAhead; n++) {
            mbar_init(&sm.tile_full[n], 1);
            mbar_init(&sm.tile_empty[n], kMmaSumWarps + kMmaOperandWarps + (rank & 1u ? 2u : 1u));  // and the issuing warp or both relays
        }
        mbar_init(&sm.drain, 1);
        sm.abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < kMmaRing * kMmaMarkWords) (&sm.again[0][0])[threadIdx.x] = 0u;
    if (warp == kIssueWarp) tmem_alloc<true>(&sm.tmem, 512);
    tmem_fence_before();
    __syncthreads();
    // (the warps that set the shared memory up also publish it)
    if (warp < kMmaSumWarps) cluster_arrive();
    else cluster_arrive_relaxed();
    if (!a.beside) grid_dependency_wait();
    if (a.before_next) grid_dependency_launch();
    MmaPlan plan;
    plan.tile = blockIdx.x / (2u * (unsigned)a.splits);
    plan.prob = 0;
    // (a lone launch has few tiles: its first one is planned before the other warps look at the order of the columns)
    bool more = true;
    if (!TABLE && warp == kPlanWarp) more = mma_plan_tile<TABLE, CHECK>(sm, a, rank, lane, plan, 0u);
    cluster_wait();
    tmem_fence_after();
    bool ok = true, done = false;
    if constexpr (CHECK) {
        int2 *stage = sm.gather + warp * 32;
        if constexpr (TABLE) {
            for (int i = threadIdx.x; i < (a.count + 31) / 32; i += kMmaThreads) sm.unsorted[i] = 0u;
            __syncthreads();
            for (int i = warp; i < a.count; i += kMmaThreads / 32)
                if (!mma_looks_sorted(a.problems[i], lane) && lane == 0) atomicOr(&sm.unsorted[i >> 5], 1u << (i & 31));
            __syncthreads();
            for (int w = 0; w < (a.count + 31) / 32; w++)
                for (unsigned m = sm.unsorted[w]; m; m &= m - 1u) mma_gather<WIDE ? 4 : 1>(a.problems[32 * w + __ffs(m) - 1], stage, warp, lane);
            __syncthreads();
        } else {
            done = !mma_looks_sorted(a.one, lane);
            if (done) mma_gather<WIDE ? 4 : 1>(a.one, stage, warp, lane);
        }
    }
    if (done) {
        // nothing left to do
    } else if (warp < kMmaSumWarps) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kMmaRegsSum));
        ok = mma_sums<TABLE>(sm, a, rank, warp, lane);
    } else if (warp < kIssueWarp) {
        if (kMmaRegsOperand != kMmaRegsLaunch) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kMmaRegsOperand));
        ok = mma_operands<TABLE, WIDE, DEEP, CHECK>(sm, a, rank, warp - kMmaSumWarps, lane);
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kMmaRegsIssue));
        if (warp == kPlanWarp && more) ok = mma_plan<TABLE, CHECK>(sm, a, rank, lane, plan, TABLE ? 0u : 1u);
        if (warp == kIssueWarp && (rank & 1u) == 0u) {
            const bool issuer = elect_one();
            ok = mma_issue(sm, rank, issuer, lane);
            if (!ok && issuer) {  // multiplies in flight get a bounded chance to end before the tensor memory is freed
                mma_commit<true>(&sm.drain, 1u << rank);
                (void)mbar_wait(&sm.drain, 0u);
            }
        }
        if (warp <= kIssueWarp + 1 && (rank & 1u) && lane == 0) ok = mma_relay(sm, rank, warp != kIssueWarp);
    }
    if (!ok) {
        *(volatile int *)&sm.abort = 1;
        *(volatile int *)a.error = 1;
    }
    __syncwarp();
    if (a.splits > 1 && !done) {
        cluster_arrive();
        cluster_wait();
        if (warp < kMmaSumWarps && *(volatile int *)&sm.abort == 0) mma_combine<TABLE>(sm, a, rank, warp, lane);
    }
    // no block leaves while another one of its cluster may still read its memory or arrive on its barriers
    tmem_fence_before();
    cluster_arrive_relaxed();
    cluster_wait();
    if (warp == kIssueWarp) tmem_free<true>(sm.tmem, 512);
    if (a.beside) grid_dependency_wait();
}

}  // namespace dlspm
