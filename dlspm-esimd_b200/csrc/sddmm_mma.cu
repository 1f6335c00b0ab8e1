// Host side of the tensor-core SDDMM (sddmm_mma.cuh): launches for one pattern and for a table of problems.
#include <algorithm>

#include "common.cuh"
#include "sddmm_mma.cuh"

using namespace dlspm;

namespace {

template <bool TABLE, bool WIDE>
int pick_launch(dlspm_ctx *ctx, const PickArgs &a, cudaStream_t st)
{
    auto kernel = sddmm_mma_kernel<TABLE, WIDE>;
    DLSPM_CUDA_TRY(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPickSmemBytes));
    const int pairs = (int)std::min<long long>(a.strips, ctx->sm_count / 2);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(2 * pairs));
    cfg.blockDim = dim3(kPickThreads);
    cfg.dynamicSmemBytes = kPickSmemBytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    DLSPM_CUDA_TRY(ctx, cudaLaunchKernelEx(&cfg, kernel, a));
    return DLSPM_OK;
}

// Byte offsets into the operands are 32-bit in the kernel (and run up to a strip past the end).
bool pick_fits(int M, int K, int N) { return ((double)std::max(M, K) + 512) * N < 1e9; }

// Microseconds of a tile of `rows` rows: its steps of 64 (conversions of rhs, whatever the rows), or the look-ups.
// Measured per tile of 112 rows: inner dimension 256 7.3 us at 2 and at 10 % nonzeros; 64 5.6 us at 10 %, 10.5 at 30 %.
double pick_tile_us(int N, int rows, double density)
{
    return std::max(1.85 * dlspm_ceil_div(N, kPickInner), (4.5 + 20.0 * density) * rows / 128.0);
}

// The strips of a pattern on its own: rows per strip and parts of a strip so that the rounds of strips over the pairs
// of blocks end together.  Returns the estimated microseconds.
double pick_shape(const dlspm_ctx *ctx, int M, int K, int N, double density, int &strip_rows, int &parts)
{
    const int pairs = ctx->sm_count / 2, tiles = dlspm_ceil_div(K, 2 * kPickCols);
    double best = 1e30;
    for (int rows = 128; rows >= 32; rows -= 16) {
        const double tile_us = pick_tile_us(N, rows, density);
        for (int s = 1; s <= 2 && s <= tiles; s++) {
            const long long strips = (long long)dlspm_ceil_div(M, rows) * s;
            const double us = (double)((strips + pairs - 1) / pairs) * (dlspm_ceil_div(tiles, s) * tile_us + 3.0 + 2.0 * (s - 1));
            if (us < best - 1e-9) {
                best = us;
                strip_rows = rows;
                parts = s;
            }
        }
    }
    return best;
}

// A problem of a grouped call: microseconds of one of its strips and of all of them on 74 pairs of blocks.  Long strips
// are cut into up to four parts, so that no pair of blocks is left with one at the end.
struct PickCost {
    int parts;
    double strip_us, all_us, gather_us;
};

PickCost pick_cost(const dlspm_sddmm_problem &q)
{
    const double whole = dlspm_ceil_div(q.K, 2 * kPickCols) * pick_tile_us(q.N, 2 * kPickRows, (double)q.nnz / ((double)q.M * q.K));
    PickCost c;
    c.parts = std::max(1, std::min({4, dlspm_ceil_div(q.K, 2 * kPickCols), (int)(whole / 60.0) + 1}));
    c.strip_us = whole / c.parts + 3.0 + 2.0 * c.parts;
    c.all_us = (double)dlspm_ceil_div(q.M, 2 * kPickRows) * c.parts * c.strip_us / 74.0;
    c.gather_us = 2.0 * q.nnz * q.N / 7.3e6;
    return c;
}

size_t pick_starts_offset(int count) { return (sizeof(PickProblem) * (size_t)count + 255) & ~(size_t)255; }

}  // namespace

// Which problems of a grouped call the tensor cores are faster for, against 7.3 TFLOP/s of the gather kernels; none of
// them where they are too few to fill the device.  Problems of up to three strips stay with the gather kernels.
void dlspm_sddmm_mma_choose(int count, const dlspm_sddmm_problem *problems, unsigned char *chosen)
{
    double all = 0.0, longest = 0.0, gather = 0.0;
    for (int i = 0; i < count; i++) {
        const dlspm_sddmm_problem &q = problems[i];
        chosen[i] = 0;
        if (q.nnz == 0 || q.M <= 3 * 2 * kPickRows || q.N <= 0 || dlspm_vec_width(q.N, q.lhs, q.rhs) != 4 || !pick_fits(q.M, q.K, q.N)) continue;
        const PickCost c = pick_cost(q);
        if (c.all_us >= 0.8 * c.gather_us) continue;
        chosen[i] = 1;
        all += c.all_us;
        gather += c.gather_us;
        longest = std::max(longest, c.strip_us);
    }
    if (count > kPickCheckMost || all + 0.5 * longest + 10.0 >= 0.8 * gather) std::fill(chosen, chosen + count, (unsigned char)0);
}

// A pattern on its own, against 4 us and 8 TFLOP/s (3 without 16-byte loads).  Measured, gather / tensor cores in us:
// 8192 x 4096, inner dimension 256, at 10 % 180 / 130, at 2 % 39 / 127; 1024 x 4096, 256, at 50 % 104 / 80; 2048 x 512,
// 256, at 50 % 32 / 23; 8192 x 8192, 64, at 10 % 92 / 188.
bool dlspm_sddmm_mma_pays_alone(const dlspm_ctx *ctx, int M, int K, int N, int nnz, int vec)
{
    if (nnz == 0 || M <= 3 * 2 * kPickRows || !pick_fits(M, K, N)) return false;
    int rows = 0, parts = 0;
    const double mma_us = 8.0 + pick_shape(ctx, M, K, N, (double)nnz / ((double)M * K), rows, parts);
    return mma_us < 0.8 * (4.0 + 2.0 * nnz * N / (vec == 4 ? 8e6 : 3e6));
}

int dlspm_sddmm_mma(dlspm_ctx *ctx, int M, int K, int N, int nnz, const int *row_offsets, const int *cols, const float *mask,
                    const float *lhs, const float *rhs, float *out, cudaStream_t st)
{
    const int rc = dlspm_mma_check(ctx);
    if (rc) return rc;
    PickArgs a = {};
    a.one = PickProblem{row_offsets, cols, lhs, rhs, mask, out, M, K, N, 0, 0, 0};
    pick_shape(ctx, M, K, N, (double)nnz / ((double)M * K), a.one.strip_rows, a.one.parts);
    a.one.strips = dlspm_ceil_div(M, a.one.strip_rows);
    a.strips = (long long)a.one.strips * a.one.parts;
    a.error = ctx->mma_error;
    if (dlspm_vec_width(N, lhs, rhs) == 4) return pick_launch<false, true>(ctx, a, st);
    return pick_launch<false, false>(ctx, a, st);
}

size_t dlspm_sddmm_mma_table_bytes(int count) { return pick_starts_offset(count) + sizeof(long long) * ((size_t)count + 1); }

long long dlspm_sddmm_mma_tables(int count, const dlspm_sddmm_problem *problems, void *image)
{
    PickProblem *tab = (PickProblem *)image;
    long long *starts = (long long *)((char *)image + pick_starts_offset(count));
    for (int i = 0; i < count; i++) {
        const dlspm_sddmm_problem &q = problems[i];
        const int strips = dlspm_ceil_div(q.M, 2 * kPickRows), rows = dlspm_ceil_div(dlspm_ceil_div(q.M, strips), 16) * 16;
        tab[i] = PickProblem{q.row_offsets, q.column_indices, q.lhs, q.rhs, q.mask_values, q.out_values, q.M, q.K, q.N, rows,
                             dlspm_ceil_div(q.M, rows), pick_cost(q).parts};
    }
    // the longest strips first: they are dealt to the pairs of blocks in turn
    std::stable_sort(tab, tab + count, [](const PickProblem &x, const PickProblem &y) {
        return (double)x.K / x.parts * (x.N + kPickInner) > (double)y.K / y.parts * (y.N + kPickInner);
    });
    long long run = 0;
    for (int i = 0; i < count; i++) {
        starts[i] = run;
        run += (long long)tab[i].strips * tab[i].parts;
    }
    starts[count] = run;
    return run;
}

int dlspm_sddmm_mma_launch_tables(dlspm_ctx *ctx, const void *tables, int count, long long strips, cudaStream_t st)
{
    const int rc = dlspm_mma_check(ctx);
    if (rc) return rc;
    PickArgs a = {};
    a.problems = (const PickProblem *)tables;
    a.strip_start = (const long long *)((const char *)tables + pick_starts_offset(count));
    a.count = count;
    a.strips = strips;
    a.error = ctx->mma_error;
    return pick_launch<true, true>(ctx, a, st);
}
