// Host side of the tensor-core SpMM (spmm_mma.cuh): launches for one matrix and for a table of problems.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "spmm_mma.cuh"

using namespace dlspm;

namespace {

template <bool TABLE, bool WIDE, bool DEEP, bool CHECK>
int mma_launch(dlspm_ctx *ctx, const MmaArgs &a, int clusters, cudaStream_t st)
{
    auto kernel = spmm_mma_kernel<TABLE, WIDE, DEEP, CHECK>;
    DLSPM_CUDA_TRY(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMmaSmemBytes));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(clusters * 2 * a.splits));
    cfg.blockDim = dim3(kMmaThreads);
    cfg.dynamicSmemBytes = kMmaSmemBytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)(2 * a.splits);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    DLSPM_CUDA_TRY(ctx, cudaLaunchKernelEx(&cfg, kernel, a));
    return DLSPM_OK;
}

void mma_shape(MmaProblem &p, int nnz)
{
    p.row_blocks = dlspm_ceil_div(p.M, 2 * kMmaRows);
    p.block_rows = dlspm_ceil_div(dlspm_ceil_div(p.M, p.row_blocks), 16) * 16;
    p.row_blocks = dlspm_ceil_div(p.M, p.block_rows);
    // the entries per chunk of a row a third longer than the mean, plus twice their spread: a row with more fetches
    // them in the chunk itself, one exposed latency for every eight (50 % nonzeros with 40 % spread of the row lengths,
    // 32 instead of 64 entries ahead: 3.3 instead of 2.8 us per chunk)
    const double mean = (double)kMmaChunk * nnz / ((double)p.M * p.K);
    p.depth = std::min(8, (int)((1.3 * mean + 2.0 * sqrt(mean)) / 8.0) + 1);
}

MmaProblem mma_problem(const dlspm_problem &q)
{
    MmaProblem p{q.values, q.row_offsets, q.column_indices, q.B, q.C, q.M, q.K, q.N, 0, 0, 0};
    mma_shape(p, q.nnz);
    return p;
}

long long mma_tiles(const MmaProblem &p) { return (long long)p.row_blocks * dlspm_ceil_div(p.N, 2 * kMmaCols); }

size_t mma_starts_offset(int count) { return (sizeof(MmaProblem) * (size_t)count + 255) & ~(size_t)255; }

// Parts of K for a launch of `tiles` tiles: as long as every part gets a pair of blocks of its own and eight chunks.
int mma_splits(const dlspm_ctx *ctx, long long tiles, int K)
{
    int s = 1;
    while (s < 4 && tiles * 4 * s <= ctx->sm_count && dlspm_ceil_div(K, kMmaChunk) >= 8 * s) s *= 2;
    return s;
}

}  // namespace

// Byte offsets into the CSR arrays (up to two chunks past the end) and the step from request to request of B, four rows, are
// 32-bit in the kernel.  B itself is addressed by 64-bit pointers; beyond 1e9 elements the kernel is not measured, and such
// problems stay with the row-gather kernels.
bool dlspm_spmm_mma_fits(int K, int N, int nnz)
{
    return ((double)K + 4 * kMmaChunk) * N < 1e9 && nnz < 1000000000;
}

// Which problems of a batch the tensor cores are faster for: chosen[i], not 0 on entry where problem i may go there, becomes
// its depth or 0.  The constants are of a build that took 1.5 us per chunk of 64 columns, more with more entries to scatter,
// and 3 us per tile; the present one takes 1.4 us per chunk at 10 % nonzeros and 1.9 at 50 % with 64 chunks a tile, tile
// included (1.7 and 2.3 with eight chunks), so the estimate leaves problems near the line to the row-gather kernel (10 to 15
// TFLOP/s).  Measured on batches of one shape with N = 3136, row-gather / tensor cores in TFLOP/s: 1024 x 4096 at 50 %
// nonzeros 15.1 / 75.6, at 10 % 11.9 / 20.4, at 5 % 10.9 / 11.5 (left to the gather), at 2 % 10.2 / 4.9; 2048 x 512 at 50 %
// 14.6 / 64.7, at 10 % 11.5 / 16.9, at 5 % 11.1 / 8.9; 512 x 2048 at 5 % 11.1 / 10.9; 256 x 256 at 20 % 11.4 / 23.6, at 10 %
// 10.6 / 12.9 (left to the gather), at 5 % 8.5 / 6.7.  A batch whose tiles are too few for the 74 pairs of blocks takes as
// long as its longest tile: then none is chosen.
void dlspm_spmm_mma_choose(int count, const dlspm_problem *problems, unsigned char *chosen)
{
    double all = 0.0, longest = 0.0, gather = 0.0;
    for (int i = 0; i < count; i++) {
        if (!chosen[i]) continue;
        chosen[i] = 0;
        const dlspm_problem &q = problems[i];
        if (q.nnz == 0 || q.M <= 0 || q.N <= 0 || q.K <= 0 || !dlspm_spmm_mma_fits(q.K, q.N, q.nnz)) continue;
        const double density = (double)q.nnz / ((double)q.M * q.K);
        const double tiles = (double)dlspm_ceil_div(q.M, 2 * kMmaRows) * dlspm_ceil_div(q.N, 2 * kMmaCols);
        const double tile_us = dlspm_ceil_div(q.K, kMmaChunk) * (1.5 + 2.4 * density) + 3.0;
        const double gather_us = 2.0 * q.nnz * q.N / 11e6;
        if (tiles * tile_us / 74.0 >= gather_us) continue;
        chosen[i] = (unsigned char)mma_problem(q).depth;
        all += tiles * tile_us / 74.0;
        longest = std::max(longest, tile_us);
        gather += gather_us;
    }
    if (count > kMmaCheckMost || std::max(all, longest) + 0.3 * longest + 8.0 >= 0.9 * gather) std::fill(chosen, chosen + count, (unsigned char)0);
}

// A matrix on its own: launch and first chunk 8.5 us, then 1.25 us per chunk and round of tiles; the row-gather
// kernels 4 us and about 9.5, 6 or 3 TFLOP/s for rows of B that allow 16-, 8- or 4-byte loads, which is what they did before
// they issued a batch's loads together.  Measured (launches in a graph), row-gather / tensor cores in us: 8192 x 2048 at 10 %,
// N = 256 74 / 52; 1024 x 4096 at 10 %, N = 1024 84 / 56, at 50 %, N = 3136 1276 / 298; 4096 x 4096 at 10 %, N = 256 85 / 57;
// 1000 x 2000 at 20 %, N = 301 65 / 55; 512 x 2048 at 30 %, N = 256 24.3 / 25.0.  Near the line the tensor cores are the
// slower way now (1024 x 1024 at 30 %, N = 512 34 / 41, 2048 x 2048 at 20 %, N = 200 43 / 55); the line stays where it was, since
// sums there are three times as close to those in 64 bits as the gather's.
bool dlspm_spmm_mma_pays_alone(const dlspm_ctx *ctx, int M, int K, int N, int nnz, int vec)
{
    if (nnz == 0 || N < 32 || !dlspm_spmm_mma_fits(K, N, nnz)) return false;
    const double density = (double)nnz / ((double)M * K);
    const long long tiles = (long long)dlspm_ceil_div(M, 2 * kMmaRows) * dlspm_ceil_div(N, 2 * kMmaCols);
    const int splits = mma_splits(ctx, tiles, K);
    const double rounds = splits > 1 ? 1.0 : (double)((tiles + ctx->sm_count / 2 - 1) / (ctx->sm_count / 2));
    const double mma_us = 8.5 + rounds * (dlspm_ceil_div(dlspm_ceil_div(K, kMmaChunk), splits) * (1.25 + 1.6 * density) + 2.5);
    const double gather_us = 4.0 + 2.0 * nnz * N / (vec == 4 ? 9.5e6 : vec == 2 ? 6e6 : 3e6);
    return mma_us < 0.9 * gather_us;
}

size_t dlspm_spmm_mma_table_bytes(int count) { return mma_starts_offset(count) + sizeof(long long) * ((size_t)count + 2); }

static_assert(sizeof(MmaProblem) == kMmaEntryBytes, "size of a table entry in common.cuh");

long long dlspm_spmm_mma_entry(const dlspm_problem &q, void *at)
{
    const MmaProblem p = mma_problem(q);
    memcpy(at, &p, sizeof(p));
    return mma_tiles(p);
}

bool dlspm_spmm_mma_deep(int depth) { return depth > kMmaDepth; }

dlspm_mma_parts dlspm_spmm_mma_tables(int count, const dlspm_problem *problems, void *image)
{
    MmaProblem *tab = (MmaProblem *)image;
    long long *starts = (long long *)((char *)image + mma_starts_offset(count));
    // The problems of the deep build first.  A tile costs about ceil(K / 64) equal steps; with the longest first the
    // fixed deal of tiles to clusters (cluster c takes tiles c, c + clusters, ...) hands every cluster the same mix.
    for (int i = 0; i < count; i++) tab[i] = mma_problem(problems[i]);
    std::stable_sort(tab, tab + count, [](const MmaProblem &x, const MmaProblem &y) {
        const bool dx = x.depth > kMmaDepth, dy = y.depth > kMmaDepth;
        return dx != dy ? dx : x.K != y.K ? x.K > y.K : x.depth > y.depth;
    });
    dlspm_mma_parts parts = {0, 0, 0, 0};
    for (int i = 0; i < count; i++) (tab[i].depth > kMmaDepth ? parts.deep : parts.rest)++;
    for (int i = 0; i < parts.deep; i++) {
        *starts++ = parts.deep_tiles;
        parts.deep_tiles += mma_tiles(tab[i]);
    }
    *starts++ = parts.deep_tiles;
    for (int i = parts.deep; i < count; i++) {
        *starts++ = parts.rest_tiles;
        parts.rest_tiles += mma_tiles(tab[i]);
    }
    *starts = parts.rest_tiles;
    return parts;
}

int dlspm_spmm_mma_launch_tables(dlspm_ctx *ctx, const void *tables, const dlspm_mma_parts &parts, bool sorted, int *error,
                                 cudaStream_t st)
{
    const int count = parts.deep + parts.rest;
    return dlspm_spmm_mma_launch_at(ctx, tables, (const long long *)((const char *)tables + mma_starts_offset(count)), parts, sorted, error, st);
}

int dlspm_spmm_mma_launch_at(dlspm_ctx *ctx, const void *tables, const long long *starts, const dlspm_mma_parts &parts, bool sorted,
                             int *error, cudaStream_t st)
{
    MmaArgs a = {};
    a.splits = 1;
    a.error = error;
    if (parts.deep) {
        a.problems = (const MmaProblem *)tables;
        a.tile_start = starts;
        a.count = parts.deep;
        a.tiles = parts.deep_tiles;
        a.before_next = parts.rest ? 1 : 0;
        const int clusters = (int)std::min<long long>(a.tiles, ctx->sm_count / 2);
        const int rc = sorted ? mma_launch<true, true, true, false>(ctx, a, clusters, st) : mma_launch<true, true, true, true>(ctx, a, clusters, st);
        if (rc) return rc;
    }
    if (parts.rest) {
        a.problems = (const MmaProblem *)tables + parts.deep;
        a.tile_start = starts + parts.deep + 1;
        a.count = parts.rest;
        a.tiles = parts.rest_tiles;
        a.before_next = 0;
        a.beside = parts.deep ? 1 : 0;
        const int clusters = (int)std::min<long long>(a.tiles, ctx->sm_count / 2);
        return sorted ? mma_launch<true, true, false, false>(ctx, a, clusters, st) : mma_launch<true, true, false, true>(ctx, a, clusters, st);
    }
    return DLSPM_OK;
}

int dlspm_spmm_mma(dlspm_ctx *ctx, int M, int K, int N, int nnz, const float *values, const int *row_offsets, const int *cols,
                   const float *B, float *C, cudaStream_t st)
{
    const int rc = dlspm_mma_check(ctx);
    if (rc) return rc;
    MmaArgs a = {};
    a.one = mma_problem(dlspm_problem{M, K, N, nnz, values, row_offsets, cols, B, C});
    a.tiles = mma_tiles(a.one);
    a.error = ctx->mma_error;
    a.splits = mma_splits(ctx, a.tiles, K);
    const int clusters = a.splits > 1 ? (int)a.tiles : (int)std::min<long long>(a.tiles, ctx->sm_count / 2);
    const bool wide = dlspm_vec_width(N, B, B) == 4, deep = a.one.depth > kMmaDepth;
    if (wide) return deep ? mma_launch<false, true, true, true>(ctx, a, clusters, st) : mma_launch<false, true, false, true>(ctx, a, clusters, st);
    return deep ? mma_launch<false, false, true, true>(ctx, a, clusters, st) : mma_launch<false, false, false, true>(ctx, a, clusters, st);
}
