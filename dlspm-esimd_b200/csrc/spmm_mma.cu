// Host side of the tensor-core SpMM (spmm_mma.cuh): launches for one matrix and for a table of problems.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "spmm_mma.cuh"

using namespace dlspm;

namespace {

template <bool TABLE, bool WIDE>
int mma_launch(dlspm_ctx *ctx, const MmaArgs &a, int clusters, cudaStream_t st)
{
    auto kernel = spmm_mma_kernel<TABLE, WIDE>;
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
    // the mean of a row's entries per chunk plus twice its spread
    const double mean = (double)kMmaChunk * nnz / ((double)p.M * p.K);
    p.depth = std::min(4, (int)((mean + 2.0 * sqrt(mean) + 1.0) / 8.0) + 1);
}

MmaProblem mma_problem(const dlspm_problem &q)
{
    MmaProblem p{q.values, q.row_offsets, q.column_indices, q.B, q.C, q.M, q.K, q.N, 0, 0, 0};
    mma_shape(p, q.nnz);
    return p;
}

long long mma_tiles(const MmaProblem &p) { return (long long)p.row_blocks * dlspm_ceil_div(p.N, 2 * kMmaCols); }

size_t mma_starts_offset(int count) { return (sizeof(MmaProblem) * (size_t)count + 255) & ~(size_t)255; }

// Byte offsets into B and into the CSR arrays are 32-bit in the kernel (and run up to two chunks past the end).
bool mma_fits(int K, int N, int nnz)
{
    return ((double)K + 4 * kMmaChunk) * N < 1e9 && nnz < 1000000000;
}

// Parts of K for a launch of `tiles` tiles: as long as every part gets a pair of blocks of its own and eight chunks.
int mma_splits(const dlspm_ctx *ctx, long long tiles, int K)
{
    int s = 1;
    while (s < 4 && tiles * 4 * s <= ctx->sm_count && dlspm_ceil_div(K, kMmaChunk) >= 8 * s) s *= 2;
    return s;
}

}  // namespace

// One of many problems of a batch: a pair of blocks needs 1.5 us per chunk of 64 columns, more with more entries to
// scatter, and 3 us per tile; the row-gather kernel 9 to 12 TFLOP/s.  Measured on batches of one shape with N = 3136,
// row-gather / tensor cores in TFLOP/s: 1024 x 4096 at 50 % nonzeros 11 / 44, at 10 % 9.3 / 17, at 5 % equal;
// 2048 x 512 at 50 % 13.5 / 45, at 10 % 11.4 / 13.1; 256 x 256 at 20 % 9.2 / 13.7, at 10 % equal.
bool dlspm_spmm_mma_pays(int M, int K, int N, int nnz)
{
    if (!mma_fits(K, N, nnz)) return false;
    const double density = (double)nnz / ((double)M * K);
    const double tiles = (double)dlspm_ceil_div(M, 2 * kMmaRows) * dlspm_ceil_div(N, 2 * kMmaCols);
    const double mma_us = tiles * (dlspm_ceil_div(K, kMmaChunk) * (1.5 + 3.2 * density) + 3.0) / 74.0;
    return mma_us < 2.0 * nnz * N / 11e6;
}

// A matrix on its own: launch and first chunk 8.5 us, then 1.25 us per chunk and round of tiles; the row-gather
// kernels 4 us and about 9.5, 6 or 3 TFLOP/s for rows of B that allow 16-, 8- or 4-byte loads.  Measured,
// row-gather / tensor cores in us: 8192 x 2048 at 10 %, N = 256 90 / 53; 1024 x 4096 at 10 %, N = 1024 101 / 57, at
// 50 %, N = 3136 1012 / 243; 512 x 2048 at 30 %, N = 256 equal; 256 x 512, N = 256 7.3 / 18.
bool dlspm_spmm_mma_pays_alone(const dlspm_ctx *ctx, int M, int K, int N, int nnz, int vec)
{
    if (nnz == 0 || N < 32 || !mma_fits(K, N, nnz)) return false;
    const double density = (double)nnz / ((double)M * K);
    const long long tiles = (long long)dlspm_ceil_div(M, 2 * kMmaRows) * dlspm_ceil_div(N, 2 * kMmaCols);
    const int splits = mma_splits(ctx, tiles, K);
    const double rounds = splits > 1 ? 1.0 : (double)((tiles + ctx->sm_count / 2 - 1) / (ctx->sm_count / 2));
    const double mma_us = 8.5 + rounds * (dlspm_ceil_div(dlspm_ceil_div(K, kMmaChunk), splits) * (1.25 + 1.6 * density) + 2.5);
    const double gather_us = 4.0 + 2.0 * nnz * N / (vec == 4 ? 9.5e6 : vec == 2 ? 6e6 : 3e6);
    return mma_us < 0.9 * gather_us;
}

size_t dlspm_spmm_mma_table_bytes(int count) { return mma_starts_offset(count) + sizeof(long long) * ((size_t)count + 1); }

long long dlspm_spmm_mma_tables(int count, const dlspm_problem *problems, void *image)
{
    MmaProblem *tab = (MmaProblem *)image;
    long long *starts = (long long *)((char *)image + mma_starts_offset(count));
    // A tile costs about ceil(K / 64) equal steps; with the longest first the fixed deal of tiles to clusters (cluster
    // c takes tiles c, c + clusters, ...) hands every cluster the same mix.
    for (int i = 0; i < count; i++) tab[i] = mma_problem(problems[i]);
    std::stable_sort(tab, tab + count, [](const MmaProblem &x, const MmaProblem &y) {
        return x.K != y.K ? x.K > y.K : x.depth > y.depth;
    });
    long long run = 0;
    for (int i = 0; i < count; i++) {
        starts[i] = run;
        run += mma_tiles(tab[i]);
    }
    starts[count] = run;
    return run;
}

int dlspm_spmm_mma_launch_tables(dlspm_ctx *ctx, const void *tables, int count, long long tiles, int *error, cudaStream_t st)
{
    MmaArgs a = {};
    a.problems = (const MmaProblem *)tables;
    a.tile_start = (const long long *)((const char *)tables + mma_starts_offset(count));
    a.count = count;
    a.splits = 1;
    a.tiles = tiles;
    a.error = error;
    return mma_launch<true, true>(ctx, a, (int)std::min<long long>(tiles, ctx->sm_count / 2), st);
}

int dlspm_spmm_mma(dlspm_ctx *ctx, int M, int K, int N, int nnz, const float *values, const int *row_offsets, const int *cols,
                   const float *B, float *C, cudaStream_t st)
{
    if (*(volatile int *)ctx->mma_error) {  // of an earlier launch
        *(volatile int *)ctx->mma_error = 0;
        return DLSPM_ERR_TIMEOUT;
    }
    MmaArgs a = {};
    a.one = mma_problem(dlspm_problem{M, K, N, nnz, values, row_offsets, cols, B, C});
    a.tiles = mma_tiles(a.one);
    a.error = ctx->mma_error;
    a.splits = mma_splits(ctx, a.tiles, K);
    const int clusters = a.splits > 1 ? (int)a.tiles : (int)std::min<long long>(a.tiles, ctx->sm_count / 2);
    if (dlspm_vec_width(N, B, B) == 4) return mma_launch<false, true>(ctx, a, clusters, st);
    return mma_launch<false, false>(ctx, a, clusters, st);
}
