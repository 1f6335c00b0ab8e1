// Host side of the tensor-core SDDMM (sddmm_mma.cuh): launches for one pattern and for a table of problems.
#include <algorithm>
#include <vector>

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

SddmmSizes sizes_of(const dlspm_sddmm_problem &q)
{
    return SddmmSizes{q.M, q.K, q.N, (double)q.nnz, q.mask_values != nullptr, dlspm_vec_width(q.N, q.lhs, q.rhs) == 4};
}

size_t pick_starts_offset(int count) { return (sizeof(PickProblem) * (size_t)count + 255) & ~(size_t)255; }

}  // namespace

bool dlspm_sddmm_mma_pays_alone(const dlspm_ctx *ctx, int M, int K, int N, int nnz, bool masked, int vec)
{
    return pick_pays_alone(ctx->sm_count, SddmmSizes{M, K, N, (double)nnz, masked, vec == 4});
}

void dlspm_sddmm_mma_choose(const dlspm_ctx *ctx, int count, const dlspm_sddmm_problem *problems, unsigned char *chosen)
{
    std::vector<SddmmSizes> sizes;
    for (int i = 0; i < count; i++) sizes.push_back(sizes_of(problems[i]));
    sddmm_route_group(ctx->sm_count, sizes, chosen);
}

int dlspm_sddmm_mma(dlspm_ctx *ctx, int M, int K, int N, int nnz, const int *row_offsets, const int *cols, const float *mask,
                    const float *lhs, const float *rhs, float *out, cudaStream_t st)
{
    const int rc = dlspm_mma_check(ctx);
    if (rc) return rc;
    PickArgs a = {};
    a.one = PickProblem{row_offsets, cols, lhs, rhs, mask, out, M, K, N, 0, 0, 0};
    const bool wide = dlspm_vec_width(N, lhs, rhs) == 4;
    const PickShape shape = pick_shape(ctx->sm_count, SddmmSizes{M, K, N, (double)nnz, mask != nullptr, wide});
    a.one.strip_rows = shape.strip_rows;
    a.one.parts = shape.parts;
    a.one.strips = dlspm_ceil_div(M, a.one.strip_rows);
    a.strips = (long long)a.one.strips * a.one.parts;
    a.error = ctx->mma_error;
    return wide ? pick_launch<false, true>(ctx, a, st) : pick_launch<false, false>(ctx, a, st);
}

size_t dlspm_sddmm_mma_table_bytes(int count) { return pick_starts_offset(count) + sizeof(long long) * ((size_t)count + 1); }

long long dlspm_sddmm_mma_tables(int count, const dlspm_sddmm_problem *problems, void *image)
{
    PickProblem *tab = (PickProblem *)image;
    long long *starts = (long long *)((char *)image + pick_starts_offset(count));
    for (int i = 0; i < count; i++) {
        const dlspm_sddmm_problem &q = problems[i];
        const PickCut c = pick_cut(sizes_of(q));
        tab[i] = PickProblem{q.row_offsets, q.column_indices, q.lhs, q.rhs, q.mask_values, q.out_values, q.M, q.K, q.N, c.strip_rows,
                             c.strips, c.parts};
    }
    std::stable_sort(tab, tab + count, [](const PickProblem &x, const PickProblem &y) {
        const auto order = [](const PickProblem &p) { return (double)p.K / p.parts * (p.N + kPickInner); };  // as pick_order
        return order(x) > order(y);
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
