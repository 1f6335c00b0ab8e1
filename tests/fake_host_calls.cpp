// The host-buffer entry points (csrc/host_api.cu) over a stand-in for the CUDA runtime, on the CPU: copies are memcpy,
// the device calls do nothing, and where `give_up` is set they raise the word that a kernel raises when a bounded wait
// runs out.  Prints per call: its status when its own kernel gave up; the status of the call after it; the status and the
// number of device calls when the word was already set on entry, and the status of the call after that.
#include <cstdio>

#include HOST_API

static bool give_up = false;
static int device_calls = 0;

static int device_call(dlspm_ctx *ctx)
{
    device_calls++;
    if (give_up) *ctx->mma_error = 1;
    return DLSPM_OK;
}

extern "C" int dlspm_spmm_csr_f32(dlspm_ctx *c, int, int, int, int, const float *, const int *, const int *, const float *, float *, void *) { return device_call(c); }
extern "C" int dlspm_sddmm_csr_f32(dlspm_ctx *c, int, int, int, int, const int *, const int *, const float *, const float *, float *, void *) { return device_call(c); }
extern "C" int dlspm_fused_sddmm_spmm_f32(dlspm_ctx *c, int, int, int, int, const int *, const int *, const float *, const float *, const float *, float *, void *) { return device_call(c); }
int dlspm_spmm_batched_at(dlspm_ctx *c, int, const dlspm_problem *, void *, cudaStream_t, void *, const unsigned char *) { return device_call(c); }
int dlspm_sddmm_batched_at(dlspm_ctx *c, int, const dlspm_sddmm_problem *, void *, void *, cudaStream_t) { return device_call(c); }
int dlspm_fused_batched_at(dlspm_ctx *c, int, const dlspm_fused_problem *, void *, void *, cudaStream_t) { return device_call(c); }
void dlspm_spmm_choose_staged(dlspm_ctx *, int count, const dlspm_problem *, unsigned char *chosen) { memset(chosen, 1, (size_t)count); }
size_t dlspm_batched_table_bytes(int) { return 256; }
size_t dlspm_rows_batched_table_bytes(int) { return 256; }
int dlspm_check_input_host(dlspm_ctx *, int, int, int, int, const int *, const int *) { return DLSPM_OK; }
int dlspm_cuda_fail(dlspm_ctx *, cudaError_t, const char *) { return DLSPM_ERR_CUDA; }
static char staging[1 << 16], table[1 << 14];
int dlspm_stage_reserve(dlspm_ctx *c, size_t bytes) { c->stage = staging; return bytes <= sizeof(staging) ? DLSPM_OK : DLSPM_ERR_NOMEM; }

extern "C" {
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *, unsigned) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t) { *p = table; return cudaSuccess; }
cudaError_t cudaFreeHost(void *) { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char *, void **, unsigned long long, cudaDriverEntryPointQueryResult *) { return cudaErrorUnknown; }
}

template <typename F>
static void report(dlspm_ctx *ctx, const char *name, F call)
{
    give_up = true;
    const int own = call();
    give_up = false;
    const int after = call();
    *ctx->mma_error = 1;
    device_calls = 0;
    const int pending = call(), made = device_calls, then = call();
    printf("%s %d %d %d %d %d\n", name, own, after, pending, made, then);
}

int main()
{
    static dlspm_ctx ctx;
    static int word = 0;
    ctx.mma_error = &word;
    int ro[5] = {0, 1, 2, 3, 4}, ci[4] = {0, 1, 2, 3};
    float v[4] = {1, 2, 3, 4}, x[16] = {}, y[16] = {}, z[16] = {}, out[16];
    const dlspm_problem p = {4, 4, 4, 4, v, ro, ci, x, out};
    const dlspm_sddmm_problem s = {4, 4, 4, 4, ro, ci, nullptr, x, y, out};
    const dlspm_fused_problem f = {4, 4, 4, 4, ro, ci, x, y, z, out};
    report(&ctx, "spmm", [&] { return dlspm_spmm_csr_f32_host(&ctx, 4, 4, 4, 4, v, ro, ci, x, out); });
    report(&ctx, "sddmm", [&] { return dlspm_sddmm_csr_f32_host(&ctx, 4, 4, 4, 4, ro, ci, x, y, out); });
    report(&ctx, "fused", [&] { return dlspm_fused_sddmm_spmm_f32_host(&ctx, 4, 4, 4, 4, ro, ci, x, y, z, out); });
    report(&ctx, "spmm_batched", [&] { return dlspm_spmm_batched_f32_host(&ctx, 1, &p); });
    report(&ctx, "sddmm_batched", [&] { return dlspm_sddmm_batched_f32_host(&ctx, 1, &s); });
    report(&ctx, "fused_batched", [&] { return dlspm_fused_batched_f32_host(&ctx, 1, &f); });
    return 0;
}
