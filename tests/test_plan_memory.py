"""Device memory of plan creation, on a fake CUDA runtime with a memory of a given size.

A plan fits where its own arrays fit: the buffer that its uploads go through is given back
before the later arrays are allocated, and where it is not to be had the uploads go row by
row, with the same contents.
"""
import pytest

from tests.host_cc import run_cpp

FAKE = r"""
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
static int padded = 0, by_rows = 0;
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
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
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
int zm_strip_width() { return 64; }
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
using namespace rsgpu;

template <typename P>
static int make(P &p, const rsgpu_config &c, std::vector<rsgpu_shot> &s, std::vector<unsigned char> &image)
{
    padded = by_rows = 0;
    const int st = p.create(&c, (int)s.size(), s.data());
    if (st == RSGPU_OK) image.assign((unsigned char *)p.arena, (unsigned char *)p.arena + p.arena_bytes);
    return st;
}

// Unlimited, then in a memory of just the plan's own arrays: status, uploads of each kind, same contents.
template <typename P>
static void both(const char *name, rsgpu_config c, int ns, int nx, int ny, int nz, bool adjoint)
{
    const int l = c.lpml;
    const size_t n = (size_t)(nx + 2 * l) * (ny ? ny + 2 * l : 1) * (nz + 2 * l);
    std::mt19937 rng(1);
    std::vector<std::vector<float>> par(8, std::vector<float>(n));
    for (auto &v : par) for (auto &x : v) x = rng() / 4.0e9f;
    std::vector<rsgpu_shot> s(ns);
    for (auto &q : s) {
        q.nx = nx; q.ny = ny; q.nz = nz;
        for (int k = 0; k < 8; k++) q.model[k] = par[k].data();
    }
    std::vector<unsigned char> a, b;
    size_t own = 0;
    capacity = ~size_t(0);
    {
        P p;
        p.adjoint_steps = adjoint;
        if (make(p, c, s, a) != RSGPU_OK) exit(1);
        own = used;
        printf("%s %d %d ", name, padded, by_rows);
    }
    if (used) exit(2);
    capacity = own;
    {
        P p;
        p.adjoint_steps = adjoint;
        const int st = make(p, c, s, b);
        printf("%d %d %d %d\n", st, padded, by_rows, (int)(a == b));
    }
    if (used) exit(3);
}

int main()
{
    rsgpu_config c{};
    c.precision = RSGPU_F32_FAST;
    c.order = 8; c.nt = 10;
    c.dx = c.dy = c.dz = 10.0; c.dt = 1e-3;
    c.tile = -1;
    c.lpml = 5;
    c.physics = RSGPU_ACOUSTIC2D;
    both<Plan>("a2", c, 50, 3, 0, 7, false);      // tables larger than the staging buffer
    both<Plan>("a2", c, 2, 160, 0, 145, false);
    c.physics = RSGPU_ELASTIC3D;
    both<Plan3D>("e3", c, 2, 20, 9, 11, true);    // work arrays behind the uploads
    c.physics = RSGPU_ACOUSTIC3D;
    both<Plan3D>("a3", c, 3, 20, 9, 11, false);
}
"""


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    # what a plan's creation does not call stays unresolved
    out = run_cpp(tmp_path_factory.mktemp("plan_memory"), FAKE,
                  ["host.cpp", "host3d.cpp", "host_fused.cpp", "host_march.cpp", "host_prep.cpp"],
                  ["-O1", "-w", "-no-pie", "-Wl,--unresolved-symbols=ignore-all"])
    return [[w if k == 0 else int(w) for k, w in enumerate(row.split())] for row in out.splitlines()]


@pytest.mark.parametrize("row,uploads,staged", [(0, 150, True), (1, 6, False), (2, 16, True), (3, 12, False)])
def test_plan_fits_where_its_arrays_fit(lines, row, uploads, staged):
    # staged: the later arrays leave the room that the staging buffer needs before them
    _, padded, by_rows, status, padded2, by_rows2, same = lines[row]
    assert (padded, by_rows) == (uploads, 0)
    assert (status, same) == (0, 1)
    assert (padded2, by_rows2) == ((uploads, 0) if staged else (0, uploads))
