// A CUDA runtime and a GEMM of host memory, to run posit_rgemm's host code (csrc/capi.cu)
// without a GPU: an allocation can be made to fail (fake_fail_at), and what the "GEMM" does to C
// is to fill it with a marker.
#include <cuda_runtime_api.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include <vector>

namespace {
int g_allocs, g_fail_at, g_live;
size_t g_used, g_peak;
std::vector<std::pair<void *, size_t>> g_blocks;
} // namespace

extern "C" {
void fake_reset(int fail_at)
{
    g_allocs = 0;
    g_fail_at = fail_at;
    g_peak = g_used;
}
int fake_allocs() { return g_allocs; }
int fake_live() { return g_live; }
size_t fake_peak() { return g_peak; }

cudaError_t cudaMallocAsync(void **p, size_t bytes, cudaStream_t)
{
    if (++g_allocs == g_fail_at)
        return cudaErrorMemoryAllocation;
    *p = aligned_alloc(256, (bytes + 255) / 256 * 256);
    g_blocks.emplace_back(*p, bytes);
    ++g_live;
    g_used += bytes;
    g_peak = g_used > g_peak ? g_used : g_peak;
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t)
{
    for (auto &b : g_blocks)
        if (b.first == p) {
            g_used -= b.second;
            b = g_blocks.back();
            g_blocks.pop_back();
            break;
        }
    free(p);
    --g_live;
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t)
{
    for (size_t i = 0; i < h; ++i)
        memcpy((char *)d + i * dp, (const char *)s + i * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t)
{
    memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned)
{
    *e = (cudaEvent_t)1;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned)
{
    *s = (cudaStream_t)8;
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaFree(void *) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n)
{
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d)
{
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int)
{
    *v = a == cudaDevAttrComputeCapabilityMajor ? 10 : 1;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *p, int)
{
    *p = nullptr;
    return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
// the device code capi.cu's headers bring along is registered and never run
void **__cudaRegisterFatBinary(void *)
{
    static void *handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
} // extern "C"

namespace pg {
enum GemmRoute { GEMM_STAGED, GEMM_FUSED_64x32, GEMM_FUSED_32x32 }; // csrc/gemm.cuh
GemmRoute gemm_route(bool, bool, int m, int n, int k, const uint32_t *, int, const uint32_t *, int, const uint32_t *, int,
                     bool)
{
    return (double)m * n * k >= 1e6 ? GEMM_STAGED : GEMM_FUSED_32x32;
}
size_t gemm_workspace_bytes(int m, int n, int k) { return 8 * ((size_t)m + n) * k; }
cudaError_t gemm_launch(bool, bool, int m, int n, int k, uint32_t, const uint32_t *, int, const uint32_t *, int, uint32_t,
                        uint32_t *C, int ldc, void *ws, cudaStream_t, bool)
{
    if (gemm_route(true, true, m, n, k, nullptr, 0, nullptr, 0, nullptr, 0, true) == GEMM_STAGED)
        memset(ws, 0xAB, gemm_workspace_bytes(m, n, k));
    for (int j = 0; j < n; ++j)
        for (int i = 0; i < m; ++i)
            C[i + (size_t)j * ldc] = 0x12345678u;
    return cudaSuccess;
}
int read_device_error(bool) { return 0; }
cudaError_t scale_launch(int, int, bool, uint32_t, uint32_t, uint32_t *, int, cudaStream_t) { return cudaSuccess; }
cudaError_t convert_launch(bool, const void *, void *, size_t, cudaStream_t) { return cudaSuccess; }
void profile_enable(bool) {}
int profile_read(double *, long long *, long long *, bool) { return 0; }
size_t rgetrf_workspace_bytes(int, int, int) { return 256; }
size_t rpotrf_workspace_bytes(int, int) { return 256; }
size_t rpotrf_upper_workspace_bytes(int, int) { return 256; }
int tuned_panel_width(bool, int) { return 32; }
int solve_cluster_ctas(int, int) { return 1; }
cudaError_t rgetrf_launch(int, int, uint32_t *, int, int *, int, int *, void *, cudaStream_t) { return cudaSuccess; }
cudaError_t rpotrf_lower_launch(int, uint32_t *, int, int, int *, void *, cudaStream_t) { return cudaSuccess; }
cudaError_t rpotrf_upper_launch(int, uint32_t *, int, int, int *, void *, cudaStream_t) { return cudaSuccess; }
cudaError_t rgetrs_launch(int, int, const uint32_t *, int, const int *, uint32_t *, int, cudaStream_t) { return cudaSuccess; }
cudaError_t rgetrs_trans_launch(int, int, const uint32_t *, int, const int *, uint32_t *, int, cudaStream_t)
{
    return cudaSuccess;
}
cudaError_t rpotrs_lower_launch(int, int, const uint32_t *, int, uint32_t *, int, cudaStream_t) { return cudaSuccess; }
cudaError_t rpotrs_upper_launch(int, int, const uint32_t *, int, uint32_t *, int, cudaStream_t) { return cudaSuccess; }
} // namespace pg
