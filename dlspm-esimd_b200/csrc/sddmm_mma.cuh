// SDDMM on the tensor cores, for the denser patterns and the longer inner dimensions: the products of 128 rows of lhs
// with 256 rows of rhs are formed densely (both operands split into three bf16 parts, six products per fp32 product,
// see mma_split.cuh), and the stored entries of the pattern pick theirs from shared memory.
//
// Why: the gather kernels read a row of rhs for every entry and are bound by L2 and L1 at 7 to 9 TFLOP/s.  The dense
// products cost the same whatever the pattern, and a row of rhs is read once per 128 rows of the pattern.
//
// A tile is 256 columns of the pattern times up to 128 of its rows, computed by a PAIR of thread blocks: columns are
// the M dimension (tensor-memory lanes, 128 per block), rows the N dimension (each block converts half of them).  A
// cluster walks a strip of rows; each block of the pair goes through columns of its own, from left to right, so that
// every row of the pattern is read once, from a cursor.
//
// Roles of the 28 warps of a block:
//   8 sum warps      add finished accumulators (one per 64 of the inner dimension) to fp32 registers and put the tile
//                    into shared memory.
//   8 operand warps  convert 64 of the inner dimension of the block's 128 rows of rhs and of its half of the rows of
//                    lhs, loaded one step ahead, into one of two stages.
//   8 pick warps     read the column indices of their rows one tile ahead, look the products up and write them.
//   1 issuing warp   (of the even block); in the odd block it relays barriers.
//
// Entries that are out of order, and products that are not finite or come from numbers that cannot be split, are
// computed one by one with fp32 multiply-adds.
#pragma once
#include "mma_split.cuh"
#include "sddmm_route.h"

namespace dlspm {

constexpr int kPickStages = 2;
constexpr int kPickSumWarps = 8, kPickOperandWarps = 8, kPickWarps = 8;
constexpr int kPickThreads = (kPickSumWarps + kPickOperandWarps + kPickWarps + 4) * 32;
constexpr int kPickRhsPlane = kPickInner * kPickCols * 2, kPickLhsPlane = kPickInner * kPickRows * 2;
constexpr int kPickRegsLaunch = 72, kPickRegsSum = 96, kPickRegsOperand = 80, kPickRegsPick = 56, kPickRegsIssue = 40;
static_assert(kPickThreads * kPickRegsLaunch <= 65536 &&
                  32 * (kPickSumWarps * kPickRegsSum + kPickOperandWarps * kPickRegsOperand + kPickWarps * kPickRegsPick + 4 * kPickRegsIssue) <=
                      kPickThreads * kPickRegsLaunch,
              "register budgets exceed what the block is launched with");
constexpr uint32_t kPickSmallColumn = 256;  // tensor memory: two main accumulators, then two for the small products
constexpr int kPickRing = 16;               // tiles whose mark (numbers that cannot be split) can be alive at once

struct PickProblem {
    const int *row_offsets;
    const int *cols;
    const float *lhs;   // M x N
    const float *rhs;   // K x N
    const float *mask;  // factors of the entries, or null
    float *out;
    int M, K, N;        // N: inner dimension
    int strip_rows;     // rows of a strip, a multiple of 16 (half of them per block)
    int strips;         // ceil(M / strip_rows)
    int parts;          // every strip is cut into so many parts of its columns (at most four) for pairs of their own
};

struct PickSmem {
    unsigned char rhs[kPickStages][3][kPickRhsPlane];  // rows of 64 numbers, 128-byte swizzle
    unsigned char lhs[kPickStages][3][kPickLhsPlane];
    float tile[2 * kPickRows][kPickCols];              // products of the tile's rows with this block's columns
    int ahead[kPickWarps][2 * kPickRows / kPickWarps][32];     // column indices of the next entries of every row
    unsigned long long full[kPickStages], empty[kPickStages];  // operands written (both blocks) / multiplies done
    unsigned long long sum_full[2], sum_empty[2];              // accumulators complete / added by all sum warps
    unsigned long long tile_full[2], tile_empty[2];            // halves of `tile` written / read by all pick warps
    unsigned long long drain;                                  // multiplies still running when a wait ran out
    unsigned slow[kPickRing];                                  // the tile holds numbers that cannot be split
    unsigned unsorted[kPickCheckMost / 32];                    // problems whose columns do not ascend
    uint32_t tmem;
    int abort;
};
constexpr size_t kPickSmemBytes = sizeof(PickSmem) + 1024;  // the swizzled planes start at a 1024-byte boundary
static_assert(kPickSmemBytes <= 232448, "shared memory of a block");

// The strips (parts of strips) of one launch, of a table of problems or of one.
struct PickArgs {
    const PickProblem *problems;
    const long long *strip_start;
    int count;
    long long strips;  // with their parts
    PickProblem one;
    int *error;
};

struct PickStrip {
    long long at;
    int prob;
    const PickProblem *p;
    int row0, rows;    // first row of the strip, rows per block
    int tile0, tiles;  // this block's tiles of 128 columns
    int part;          // its part of the strip, of 2 * parts
    int chunks;
};

// First tile of part b of 2 * parts of a strip, in tiles of 128 columns.
__device__ __forceinline__ int pick_boundary(const PickProblem &p, int b)
{
    return (int)((long long)((p.K + kPickCols - 1) / kPickCols) * b / (2 * p.parts));
}

template <bool TABLE>
__device__ __forceinline__ bool pick_strip_load(PickStrip &s, const PickArgs &a, unsigned rank)
{
    if (s.at >= a.strips) return false;
    long long first = 0;
    if constexpr (TABLE) {
        int lo = s.prob, hi = a.count - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(a.strip_start + mid) <= s.at) lo = mid;
            else hi = mid - 1;
        }
        s.prob = lo;
        s.p = a.problems + lo;
        first = __ldg(a.strip_start + lo);
    } else {
        s.p = &a.one;
    }
    const int i = (int)(s.at - first), parts = s.p->parts;
    const int strip = i / parts;
    s.rows = s.p->strip_rows >> 1;
    s.row0 = strip * s.p->strip_rows;
    // both blocks walk through as many tiles as the one that has more
    const int pair = i - strip * parts, begin = pick_boundary(*s.p, 2 * pair), middle = pick_boundary(*s.p, 2 * pair + 1);
    s.part = 2 * pair + (int)(rank & 1u);
    s.tile0 = (rank & 1u) ? middle : begin;
    s.tiles = max(middle - begin, pick_boundary(*s.p, 2 * pair + 2) - middle);
    s.chunks = (s.p->N + kPickInner - 1) / kPickInner;
    return true;
}

// The same, past strips of problems that were computed at the start of the kernel.
template <bool TABLE>
__device__ __forceinline__ bool pick_strip_next(PickStrip &s, const PickArgs &a, const PickSmem &sm, unsigned rank)
{
    while (pick_strip_load<TABLE>(s, a, rank)) {
        if (!TABLE || !((sm.unsorted[s.prob >> 5] >> (s.prob & 31)) & 1u)) return true;
        s.at += gridDim.x >> 1;
    }
    return false;
}

struct PickStage {
    int stage;
    unsigned parity;
    __device__ __forceinline__ void next()
    {
        if (++stage == kPickStages) {
            stage = 0;
            parity ^= 1u;
        }
    }
};

// ---- operand warps ------------------------------------------------------------------------------------

// Pairs of rows of an operand: lanes 0..15 hold columns 4 * (lane % 16) .. + 3 of a row, lanes 16..31 of the next
// row.  `at`: byte offset of this lane's columns in its first row, `step`: of two rows, `last`: in the last row of
// the operand (rows past the end repeat it; their products are not picked).  Columns past the end are zero in lhs;
// in rhs they repeat others, which zero in lhs cancels (a product that is not finite then is computed again).
template <int PAIRS, bool WIDE, bool ZERO>
__device__ __forceinline__ void pick_load(float4 (&d)[PAIRS], const float *__restrict__ base, unsigned at, unsigned step, unsigned last, int left)
{
    const char *from = reinterpret_cast<const char *>(base);
#pragma unroll
    for (int i = 0; i < PAIRS; i++) {
        const char *src = from + min(at + i * step, last);
        if constexpr (ZERO) d[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if constexpr (WIDE) {
            if (!ZERO || left > 0) d[i] = __ldg(reinterpret_cast<const float4 *>(src));
        } else {
            const float *f = reinterpret_cast<const float *>(src);
            if (!ZERO || left > 0) d[i].x = __ldg(f);
            if (!ZERO || left > 1) d[i].y = __ldg(f + (ZERO ? 1 : min(1, left - 1)));
            if (!ZERO || left > 2) d[i].z = __ldg(f + (ZERO ? 2 : min(2, left - 1)));
            if (!ZERO || left > 3) d[i].w = __ldg(f + (ZERO ? 3 : min(3, left - 1)));
        }
    }
}

// Writes them split, the 16-byte units of row r permuted by XOR with r (mod 8); the parts are `stride` bytes apart.
template <int PAIRS>
__device__ __forceinline__ void pick_store(uint32_t plane, const float4 (&d)[PAIRS], int row, int lane, int stride, unsigned &least)
{
    float small = 1.f;
#pragma unroll
    for (int i = 0; i < PAIRS; i++) {
        const int r = row + 2 * i;
        const uint32_t at = plane + r * 128 + ((((lane & 15) >> 1) ^ (r & 7)) << 4) + (lane & 1) * 8;
        small = min3_magnitude(small, d[i].x, d[i].y);
        small = min3_magnitude(small, d[i].z, d[i].w);
        uint32_t x1, x2, x3, y1, y2, y3;
        split_pair(d[i].x, d[i].y, x1, x2, x3);
        split_pair(d[i].z, d[i].w, y1, y2, y3);
        store_shared(at, x1, y1);
        store_shared(at + stride, x2, y2);
        store_shared(at + 2 * stride, x3, y3);
    }
    if (small < kSplitSmall) {  // a zero, or a number that cannot be split
#pragma unroll
        for (int i = 0; i < PAIRS; i++) {
            least = split_magnitude(d[i].x, least);
            least = split_magnitude(d[i].y, least);
            least = split_magnitude(d[i].z, least);
            least = split_magnitude(d[i].w, least);
        }
    }
}

template <bool TABLE, bool WIDE>
__device__ __forceinline__ bool pick_operands(PickSmem &sm, const PickArgs &a, unsigned rank, int warp, int lane)
{
    volatile int *abort = &sm.abort;
    constexpr int kRhs = kPickCols / kPickOperandWarps / 2, kLhs = kPickRows / kPickOperandWarps / 2;  // pairs of rows per warp
    const int rhs_row = warp * (2 * kRhs) + (lane >> 4), lhs_row = warp * (2 * kLhs) + (lane >> 4), k = 4 * (lane & 15);
    const unsigned side = rank & 1u;
    float4 rhs[kRhs], lhs[kLhs];
    PickStrip s;
    s.at = blockIdx.x >> 1;
    s.prob = 0;
    bool have = pick_strip_next<TABLE>(s, a, sm, rank);
    int tile = 0, chunk = 0;
    auto load = [&] {
        const unsigned N = (unsigned)s.p->N;
        const int first = chunk * kPickInner + k, left = (int)N - first;  // columns from this lane's first one on
        const unsigned kr = (unsigned)min(first, WIDE ? (int)N - 4 : (int)N - 1), kl = (unsigned)min(first, (int)N - 1);
        const unsigned j = (unsigned)((s.tile0 + tile) * kPickCols + rhs_row);
        const unsigned i = (unsigned)(s.row0 + (int)side * s.rows + lhs_row);
        pick_load<kRhs, WIDE, false>(rhs, s.p->rhs, 4u * (j * N + kr), 8u * N, 4u * ((unsigned)(s.p->K - 1) * N + kr), max(left, 1));
        pick_load<kLhs, WIDE, true>(lhs, s.p->lhs, 4u * (i * N + kl), 8u * N, 4u * ((unsigned)(s.p->M - 1) * N + kl), left);
    };
    if (have) load();
    PickStage st{0, 0u};
    int ring = 0;
    unsigned least = 0xffffffffu;
    while (have) {
        if (!mbar_wait_suspended(&sm.empty[st.stage], st.parity ^ 1u, abort)) return false;
        pick_store<kRhs>(smem_u32(&sm.rhs[st.stage][0][0]), rhs, rhs_row, lane, kPickRhsPlane, least);
        pick_store<kLhs>(smem_u32(&sm.lhs[st.stage][0][0]), lhs, lhs_row, lane, kPickLhsPlane, least);
        const int now = ring;
        if (++chunk == s.chunks) {
            chunk = 0;
            ring = (ring + 1) % kPickRing;
            if (++tile == s.tiles) {
                tile = 0;
                s.at += gridDim.x >> 1;
                have = pick_strip_next<TABLE>(s, a, sm, rank);
            }
        }
        if (have) load();
        if (__any_sync(0xffffffffu, least < kSplitLeast) && lane == 0) mark_in_pair(&sm.slow[now], 1u, rank);  // rows of lhs are shared
        if (chunk == 0) least = 0xffffffffu;
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.full[st.stage]);
        st.next();
    }
    return true;
}

// ---- issuing warp (of the even block) and relay (odd block) ------------------------------------------------

template <bool TABLE>
__device__ __forceinline__ bool pick_issue(PickSmem &sm, const PickArgs &a, unsigned rank, bool issuer)
{
    volatile int *abort = &sm.abort;
    PickStrip s;
    s.at = blockIdx.x >> 1;
    s.prob = 0;
    const unsigned pair_mask = 3u << rank;
    const uint32_t tmem = sm.tmem;
    const int part_a[5] = {2, 1, 1, 0, 0}, part_b[5] = {0, 1, 0, 2, 1};  // of the five small products
    const uint64_t rhs0 = mma_descriptor(smem_u32(&sm.rhs[0][0][0]), 0, 1024, kSwizzle128);
    const uint64_t lhs0 = mma_descriptor(smem_u32(&sm.lhs[0][0][0]), 0, 1024, kSwizzle128);
    constexpr uint64_t kRhs = kPickRhsPlane >> 4, kLhs = kPickLhsPlane >> 4;
    unsigned g = 0, done = 0;  // chunks (one main accumulator each) and tiles so far
    PickStage st{0, 0u};
    while (pick_strip_next<TABLE>(s, a, sm, rank)) {
        const uint32_t instruction = mma_instruction(256, 2 * s.rows, false, false);
        for (int tile = 0; tile < s.tiles; tile++, done++) {
            const uint32_t small = tmem + kPickSmallColumn + (done & 1u) * 128u;
            for (int c = 0; c < s.chunks; c++, g++) {
                // (the accumulator of the small products was read together with its tile's last main one)
                if (g >= 2u && !mbar_wait_suspended(&sm.sum_empty[g & 1u], ((g >> 1) - 1u) & 1u, abort)) return false;
                if (!mbar_wait_suspended(&sm.full[st.stage], st.parity, abort)) return false;
                tmem_fence_after();
                const uint32_t main = tmem + (g & 1u) * 128u;
                const uint64_t rhs = rhs0 + st.stage * (3 * kRhs), lhs = lhs0 + st.stage * (3 * kLhs);
                const int steps = min(kPickInner / 16, (s.p->N - c * kPickInner + 15) / 16);
                if (issuer) {
                    for (int ks = 0; ks < steps; ks++) {
                        const uint64_t x = rhs + ks * (32 >> 4), y = lhs + ks * (32 >> 4);
#pragma unroll
                        for (int j = 0; j < 5; j++)
                            mma_bf16<true>(small, x + part_a[j] * kRhs, y + part_b[j] * kLhs, instruction, c + j + ks > 0);
                        mma_bf16<true>(main, x, y, instruction, ks > 0);
                    }
                    mma_commit<true>(&sm.empty[st.stage], pair_mask);
                    mma_commit<true>(&sm.sum_full[g & 1u], pair_mask);
                }
                __syncwarp();
                st.next();
            }
        }
        s.at += gridDim.x >> 1;
    }
    return true;
}

// Passes the odd block's barriers on to the even block's, one arrival per phase.
template <bool TABLE>
__device__ __forceinline__ bool pick_relay(PickSmem &sm, const PickArgs &a, unsigned rank, bool sums)
{
    volatile int *abort = &sm.abort;
    PickStrip s;
    s.at = blockIdx.x >> 1;
    s.prob = 0;
    const unsigned slots = sums ? 2u : (unsigned)kPickStages;
    unsigned long long *own = sums ? sm.sum_empty : sm.full;
    const uint32_t other = cluster_map(smem_u32(own), rank ^ 1u);
    unsigned g = 0;
    while (pick_strip_next<TABLE>(s, a, sm, rank)) {
        for (int c = 0; c < s.tiles * s.chunks; c++, g++) {
            if (!mbar_wait_suspended(&own[g % slots], (g / slots) & 1u, abort)) return false;
            mbar_arrive_cluster(other + (g % slots) * 8u);
        }
        s.at += gridDim.x >> 1;
    }
    return true;
}

// ---- sum warps --------------------------------------------------------------------------------------------

// Warp w: tensor-memory lanes 32 * (w % 4) .. + 31 (columns of the pattern), accumulator columns 64 * (w / 4) .. + 63
// (its rows).
template <bool TABLE>
__device__ __forceinline__ bool pick_sums(PickSmem &sm, const PickArgs &a, unsigned rank, int warp, int lane)
{
    volatile int *abort = &sm.abort;
    PickStrip s;
    s.at = blockIdx.x >> 1;
    s.prob = 0;
    const int half = (warp >> 2) * kPickRows, quarter = warp & 3;
    const uint32_t tmem = sm.tmem + ((uint32_t)quarter << 21) + (uint32_t)half;
    unsigned g = 0, done = 0;
    while (pick_strip_next<TABLE>(s, a, sm, rank)) {
        const int columns = 2 * s.rows - half;
        for (int tile = 0; tile < s.tiles; tile++, done++) {
            float acc[kPickRows];
#pragma unroll
            for (int j = 0; j < kPickRows; j++) acc[j] = 0.f;
            for (int c = 0; c < s.chunks; c++, g++) {
                if (!mbar_wait_suspended(&sm.sum_full[g & 1u], (g >> 1) & 1u, abort)) return false;
                tmem_fence_after();
                tmem_add(acc, tmem + (g & 1u) * 128u, columns);
                if (c + 1 == s.chunks) tmem_add(acc, tmem + kPickSmallColumn + (done & 1u) * 128u, columns);
                tmem_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sm.sum_empty[g & 1u]);
            }
            if (!mbar_wait_suspended(&sm.tile_empty[warp >> 2], (done & 1u) ^ 1u, abort)) return false;
            float *out = &sm.tile[half][32 * quarter + lane];
#pragma unroll
            for (int j = 0; j < kPickRows; j++) out[j * kPickCols] = acc[j];
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.tile_full[warp >> 2]);
        }
        s.at += gridDim.x >> 1;
    }
    return true;
}

// ---- pick warps -------------------------------------------------------------------------------------------

// Entries q .. of row `row`, as many as are left of four, eight lanes an entry, from the operands.
template <bool WIDE>
__device__ __forceinline__ void pick_four(const PickProblem &p, int row, int q, int left, int lane)
{
    const int e = lane >> 3;
    float sum = 0.f;
    if (e < left) {
        const float *x = p.lhs + (size_t)row * (size_t)p.N, *y = p.rhs + (size_t)__ldg(p.cols + q + e) * (size_t)p.N;
        if constexpr (WIDE) {
#pragma unroll 4
            for (int k = 4 * (lane & 7); k < p.N; k += 32) {
                const float4 a = __ldg(reinterpret_cast<const float4 *>(x + k)), b = __ldg(reinterpret_cast<const float4 *>(y + k));
                sum = fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, sum))));
            }
        } else {
#pragma unroll 4
            for (int k = lane & 7; k < p.N; k += 8) sum = fmaf(__ldg(x + k), __ldg(y + k), sum);
        }
    }
#pragma unroll
    for (int d = 4; d >= 1; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
    if (e < left && (lane & 7) == 0) p.out[q + e] = p.mask ? __ldg(p.mask + q + e) * sum : sum;
}

// First entries at or behind column `col` of the warp's rows (row r: entries start .. stop of lane r), 32 probes a
// row and the rows' probes in flight together; the result on lane r.
template <int ROWS>
__device__ __forceinline__ int pick_lower_bounds(const int *__restrict__ cols, int start, int stop, int col, int lane)
{
    int lo = start, hi = stop;
    while (__any_sync(0xffffffffu, lo < hi)) {
        int seen[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; r++) {
            const int l = __shfl_sync(0xffffffffu, lo, r), h = __shfl_sync(0xffffffffu, hi, r);
            const int at = l + lane * max(1, (h - l + 31) / 32);
            seen[r] = at < h ? __ldg(cols + at) : 0x7fffffff;
        }
#pragma unroll
        for (int r = 0; r < ROWS; r++) {
            const int below = __popc(__ballot_sync(0xffffffffu, seen[r] < col));
            if (lane == r && lo < hi) {
                const int step = max(1, (hi - lo + 31) / 32), l = lo;
                if (below > 0) lo = l + (below - 1) * step + 1;
                hi = min(hi, l + below * step);
            }
        }
    }
    return lo;
}

// Starts the copy of entry q's column index to shared memory; behind the end of the row a column that no tile has.
__device__ __forceinline__ void pick_fetch(int *to, const int *__restrict__ cols, int q, int end)
{
    if (q < end) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(to)), "l"(cols + q) : "memory");
    else *to = 0x7fffffff;
}

// Rows warp, warp + 8, .. of the strip; lane r (< 16) holds the cursor of the warp's r-th row and the end of its
// part.  Of every row 32 entries are at hand in shared memory, fetched one tile ahead (a lane reads only what it
// fetched itself).
template <bool TABLE, bool WIDE>
__device__ __forceinline__ bool pick_entries(PickSmem &sm, const PickArgs &a, unsigned rank, int warp, int lane)
{
    constexpr int kRows = 2 * kPickRows / kPickWarps, kTurn = kRows / 2;
    volatile int *abort = &sm.abort;
    int(*const ahead)[32] = sm.ahead[warp];
    PickStrip s;
    s.at = blockIdx.x >> 1;
    s.prob = 0;
    unsigned done = 0;
    while (pick_strip_next<TABLE>(s, a, sm, rank)) {
        const PickProblem &p = *s.p;
        int cursor = 0, end = 0;
        {
            const int i = warp + kPickWarps * lane, row = s.row0 + i;
            if (lane < kRows && i < 2 * s.rows && row < p.M) {
                cursor = __ldg(p.row_offsets + row);
                end = __ldg(p.row_offsets + row + 1);
            }
            // The parts' boundaries are made a rising sequence whatever the columns' order, so that every entry
            // belongs to one part.
            const int start = cursor, stop = end;
            for (int b = 1; b <= s.part + 1 && b < 2 * p.parts; b++) {
                const int at = pick_lower_bounds<kRows>(p.cols, start, stop, pick_boundary(p, b) * kPickCols, lane);
                if (b <= s.part) cursor = max(cursor, at);
                else end = max(cursor, at);
            }
        }
        for (int r = 0; r < kRows; r++)
            pick_fetch(&ahead[r][lane], p.cols, __shfl_sync(0xffffffffu, cursor, r) + lane, __shfl_sync(0xffffffffu, end, r));
        for (int tile = 0; tile < s.tiles; tile++, done++) {
            const int j0 = (s.tile0 + tile) * kPickCols;
            bool slow = false;
#pragma unroll 1
            for (int h = 0; h < 2; h++) {
                if (!mbar_wait_suspended(&sm.tile_full[h], done & 1u, abort)) return false;
                if (h == 0) {
                    slow = *(volatile unsigned *)&sm.slow[done % kPickRing] != 0u;
                    // the mark of a tile that all warps are done with, and that the operand warps do not reach yet
                    if (warp == 0 && lane == 0) sm.slow[(done + kPickRing / 2) % kPickRing] = 0u;
                }
                // Eight rows at a time, so that their chains of votes, look-ups and fetches overlap; once more while
                // a row has 32 entries and more left in the tile (the other rows then find none).
                bool more;
                do {
                    more = false;
                    asm volatile("cp.async.wait_all;" ::: "memory");
                    int q[kTurn], n[kTurn];
                    float v[kTurn], probe = 0.f;
#pragma unroll
                    for (int x = 0; x < kTurn; x++) {
                        const int r = h * kTurn + x;
                        q[x] = __shfl_sync(0xffffffffu, cursor, r) + lane;
                        // the entries at hand up to the first that does not lie in the tile
                        const unsigned d = (unsigned)(ahead[r][lane] - j0);
                        n[x] = __clz(__brev(__ballot_sync(0xffffffffu, d >= (unsigned)kPickCols)));  // 32 if none
                        v[x] = sm.tile[warp + kPickWarps * r][d & (kPickCols - 1)];
                    }
#pragma unroll
                    for (int x = 0; x < kTurn; x++)
                        if (lane < n[x]) {
                            p.out[q[x]] = p.mask ? __ldg(p.mask + q[x]) * v[x] : v[x];
                            probe = fmaf(v[x], 0.f, probe);
                        }
                    if (__any_sync(0xffffffffu, probe != 0.f) || slow) {  // NaN compares unequal
#pragma unroll 1
                        for (int x = 0; x < kTurn; x++) {
                            const int r = h * kTurn + x;
                            const int at = __shfl_sync(0xffffffffu, cursor, r);
                            const unsigned d = (unsigned)(ahead[r][lane] - j0);
                            const int count = __clz(__brev(__ballot_sync(0xffffffffu, d >= (unsigned)kPickCols)));
                            __syncwarp();
                            for (int e = 0; e < count; e += 4) pick_four<WIDE>(p, s.row0 + warp + kPickWarps * r, at + e, count - e, lane);
                        }
                    }
                    __syncwarp();
#pragma unroll
                    for (int x = 0; x < kTurn; x++) {
                        const int r = h * kTurn + x;
                        if (n[x] > 0) pick_fetch(&ahead[r][lane], p.cols, q[x] + n[x], __shfl_sync(0xffffffffu, end, r));
                        if (lane == r) cursor += n[x];
                        more = more || n[x] == 32;
                    }
                } while (more);
                __syncwarp();
                if (lane == 0) mbar_arrive(&sm.tile_empty[h]);
            }
        }
        // entries that were never reached are out of order
        for (int r = 0; r < kRows; r++) {
            const int stop = __shfl_sync(0xffffffffu, end, r);
            for (int q = __shfl_sync(0xffffffffu, cursor, r); q < stop; q += 4)
                pick_four<WIDE>(p, s.row0 + warp + kPickWarps * r, q, stop - q, lane);
        }
        s.at += gridDim.x >> 1;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    return true;
}

// ---- columns out of order ---------------------------------------------------------------------------------------

// Looks at eight entries each of 32 rows.  Entries out of order that this does not find are computed one by one; a pattern
// whose rows are out of order as a rule would take ten times as long that way as with the loop below.
__device__ __forceinline__ bool pick_looks_sorted(const PickProblem &p, int lane)
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

// A whole problem entry by entry, by all warps of the launch.
template <bool WIDE>
__device__ __forceinline__ void pick_all(const PickProblem &p, int warp, int lane)
{
    for (int row = (int)blockIdx.x * (kPickThreads / 32) + warp; row < p.M; row += (int)gridDim.x * (kPickThreads / 32)) {
        const int end = __ldg(p.row_offsets + row + 1);
        for (int q = __ldg(p.row_offsets + row); q < end; q += 4) pick_four<WIDE>(p, row, q, end - q, lane);
    }
}

// Grid: pairs of blocks; pair i takes the strips i, i + pairs, ...  error[0] is set to 1 if a bounded wait ran out.
// TABLE: strips of a table of problems, otherwise of the one among the arguments.  WIDE: rows of lhs and rhs are
// 16-byte aligned.
template <bool TABLE, bool WIDE>
__global__ void __launch_bounds__(kPickThreads, 1) sddmm_mma_kernel(const __grid_constant__ PickArgs a)
{
    extern __shared__ unsigned char smem_raw[];
    PickSmem &sm = *reinterpret_cast<PickSmem *>(smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned rank = cluster_rank();
    constexpr int kFirstPick = kPickSumWarps + kPickOperandWarps, kIssueWarp = kFirstPick + kPickWarps;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kPickStages; s++) {
            mbar_init(&sm.full[s], kPickOperandWarps + (rank & 1u ? 0u : 1u));  // even block: plus the odd one's relay
            mbar_init(&sm.empty[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(&sm.sum_full[b], 1);
            mbar_init(&sm.sum_empty[b], kPickSumWarps + (rank & 1u ? 0u : 1u));
            mbar_init(&sm.tile_full[b], kPickSumWarps / 2);
            mbar_init(&sm.tile_empty[b], kPickWarps);
        }
        mbar_init(&sm.drain, 1);
        sm.abort = 0;
        for (int i = 0; i < kPickRing; i++) sm.slow[i] = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kIssueWarp) tmem_alloc<true>(&sm.tmem, 512);
    tmem_fence_before();
    __syncthreads();
    // (the warps that set the shared memory up also publish it)
    if (warp < kPickSumWarps) cluster_arrive();
    else cluster_arrive_relaxed();
    grid_dependency_wait();
    cluster_wait();
    tmem_fence_after();
    bool ok = true, done = false;
    if constexpr (TABLE) {
        for (int i = threadIdx.x; i < (a.count + 31) / 32; i += kPickThreads) sm.unsorted[i] = 0u;
        __syncthreads();
        for (int i = warp; i < a.count; i += kPickThreads / 32)
            if (!pick_looks_sorted(a.problems[i], lane) && lane == 0) atomicOr(&sm.unsorted[i >> 5], 1u << (i & 31));
        __syncthreads();
        for (int w = 0; w < (a.count + 31) / 32; w++)
            for (unsigned m = sm.unsorted[w]; m; m &= m - 1u) pick_all<WIDE>(a.problems[32 * w + __ffs(m) - 1], warp, lane);
    } else {
        done = !pick_looks_sorted(a.one, lane);
        if (done) pick_all<WIDE>(a.one, warp, lane);
    }
    if (done) {
        // nothing left to do
    } else if (warp < kPickSumWarps) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kPickRegsSum));
        ok = pick_sums<TABLE>(sm, a, rank, warp, lane);
    } else if (warp < kFirstPick) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kPickRegsOperand));
        ok = pick_operands<TABLE, WIDE>(sm, a, rank, warp - kPickSumWarps, lane);
    } else if (warp < kIssueWarp) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kPickRegsPick));
        ok = pick_entries<TABLE, WIDE>(sm, a, rank, warp - kFirstPick, lane);
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kPickRegsIssue));
        if (warp == kIssueWarp && (rank & 1u) == 0u) {
            const bool issuer = elect_one();
            ok = pick_issue<TABLE>(sm, a, rank, issuer);
            if (!ok && issuer) {  // multiplies in flight get a bounded chance to end before the tensor memory is freed
                mma_commit<true>(&sm.drain, 1u << rank);
                (void)mbar_wait(&sm.drain, 0u);
            }
        }
        if (warp <= kIssueWarp + 1 && (rank & 1u) && lane == 0) ok = pick_relay<TABLE>(sm, a, rank, warp != kIssueWarp);
    }
    if (!ok) {
        *(volatile int *)&sm.abort = 1;
        *(volatile int *)a.error = 1;
    }
    __syncwarp();
    // no block leaves while another one of its cluster may still arrive on its barriers
    tmem_fence_before();
    cluster_arrive_relaxed();
    cluster_wait();
    if (warp == kIssueWarp) tmem_free<true>(sm.tmem, 512);
}

}  // namespace dlspm
