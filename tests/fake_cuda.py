"""A CUDA runtime in host memory, enough for the library's host files: allocations from a
device of `capacity` bytes, copies done at once, kernels left out.  What a test's calls do
not reach stays unresolved.
"""
SOURCES = ["host.cpp", "host3d.cpp", "host_fused.cpp", "host_march.cpp", "host_prep.cpp"]
FLAGS = ["-O1", "-w", "-no-pie", "-Wl,--unresolved-symbols=ignore-all"]

FAKE_CUDA = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <random>
#include <vector>
#include <cuda.h>
#include <cuda_runtime.h>
#include "rsgpu.h"
#include "rsgpu_plan.h"
#include "rsgpu_plan3d.h"
#include "rsgpu_host.h"

static size_t capacity = ~size_t(0), used = 0;
static int padded = 0, by_rows = 0, unordered = 0;
static std::map<void *, size_t> live;
static cudaStream_t const stream = (cudaStream_t)0x10;

extern "C" {
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = stream; return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *) { *p = (cudaMemPool_t)0x20; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t)
{
    if (n > capacity - used) return cudaErrorMemoryAllocation;
    *p = aligned_alloc(256, (n + 255) / 256 * 256);
    std::memset(*p, 0xa5, n);
    live[*p] = n;
    used += n;
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t)
{
    if (!live.count(p)) abort();
    used -= live[p];
    live.erase(p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind kind)
{
    // outside the order of a non-blocking stream, and from pageable memory not even done on return
    unordered += kind == cudaMemcpyHostToDevice;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t)
{
    by_rows++;
    for (size_t r = 0; r < h; r++) std::memcpy((char *)d + r * dp, (const char *)s + r * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemcpy3DAsync(const cudaMemcpy3DParms *q, cudaStream_t)
{
    by_rows++;
    for (size_t z = 0; z < q->extent.depth; z++)
        for (size_t y = 0; y < q->extent.height; y++)
            std::memcpy((char *)q->dstPtr.ptr + (z * q->dstPtr.ysize + y) * q->dstPtr.pitch,
                        (const char *)q->srcPtr.ptr + (z * q->srcPtr.ysize + y) * q->srcPtr.pitch, q->extent.width);
    return cudaSuccess;
}
static CUresult encode(...) { return CUDA_SUCCESS; }
cudaError_t cudaGetDriverEntryPoint(const char *, void **fn, unsigned long long, cudaDriverEntryPointQueryResult *q)
{
    *fn = (void *)encode;
    *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
}
namespace rsgpu {
int tile_count_2d() { return 11; }
TileShape tile_shape_2d(int) { return {32, 16, 2, 8}; }
int coef_row_stride() { return 9; }
int zm_strip_width() { return 112; }
int zm_resident_ctas(int, int) { return 296; }
int march_resident_ctas() { return 4; }
cudaError_t upload_padded(void *dst, int pitch, long long plane, const void *src, int w, int h, int d, int es, void *staging, cudaStream_t)
{
    padded++;
    if (live[staging] < (size_t)w * h * d * es) abort();
    std::memcpy(staging, src, (size_t)w * h * d * es);
    for (int z = 0; z < d; z++)
        for (int y = 0; y < h; y++)
            std::memcpy((char *)dst + ((size_t)z * plane + (size_t)y * pitch) * es,
                        (char *)staging + ((size_t)z * h + y) * w * es, (size_t)w * es);
    return cudaSuccess;
}
}
"""
