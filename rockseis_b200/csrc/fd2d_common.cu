// Dispatch of the 2D half-step kernels by precision, and the small per-step
// kernels (source injection / receiver recording, step counter).
#include "fd2d_kernels.cuh"

namespace rsgpu {


cudaError_t launch_step_2d(int prec, int cfg, int physics, int half, int flags, const void *args, const void *coefs,
                           const void *maps, int *err, int grid, cudaStream_t st)
{
    const char *v = prec == PREC_F32_EXACT ? "f32x" : prec == PREC_F32_FAST ? "f32f" : "f64";
    Launch2DFn fn = launch_2d_table(v, cfg);
    if (!fn) return cudaErrorInvalidValue;
    return fn(physics, half, flags, args, coefs, maps, err, grid, st);
}

cudaError_t launch_injrec_2d(int prec, const void *shots, const void *plans, int nshots, double dt, int it_base,
                             const int *it_dev, int threads, cudaStream_t st)
{
    if (prec == PREC_F64)
        return launch_pdl(inject_record_2d<double, MODE_IEEE>, nshots, threads, 0, st, (const Shot2D<double> *)shots,
                          (const InjRec<double> *)plans, dt, it_base, it_dev);
    return launch_pdl(prec == PREC_F32_EXACT ? inject_record_2d<float, MODE_IEEE> : inject_record_2d<float, MODE_FAST>,
                      nshots, threads, 0, st, (const Shot2D<float> *)shots, (const InjRec<float> *)plans, (float)dt,
                      it_base, it_dev);
}

// Contiguous [d][h][w] rows into a pitched, guarded array (w*h*d values).
template <typename T>
static __global__ void __launch_bounds__(256) pad_rows(T *dst, int pitch, long long plane, const T *src, int w, int h,
                                                       long long n)
{
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        const long long row = k / w;
        dst[row / h * plane + row % h * pitch + (k - row * w)] = src[k];
    }
}

cudaError_t upload_padded(void *dst, int pitch, long long plane, const void *src, int w, int h, int d, int es,
                          void *staging, cudaStream_t st)
{
    const long long n = (long long)w * h * d;
    cudaError_t e = cudaMemcpyAsync(staging, src, (size_t)n * es, cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
    const int grid = (int)((n + 255) / 256 < 4736 ? (n + 255) / 256 : 4736);   // 148 SMs x 32
    if (es == 8) pad_rows<<<grid, 256, 0, st>>>((double *)dst, pitch, plane, (const double *)staging, w, h, n);
    else pad_rows<<<grid, 256, 0, st>>>((float *)dst, pitch, plane, (const float *)staging, w, h, n);
    return cudaGetLastError();
}

cudaError_t launch_advance(int *it_dev, int by, cudaStream_t st)
{
    advance_counter<<<1, 32, 0, st>>>(it_dev, by);
    return cudaGetLastError();
}

cudaError_t launch_set_counter(int *it_dev, int value, cudaStream_t st)
{
    set_counter<<<1, 32, 0, st>>>(it_dev, value);
    return cudaGetLastError();
}

// Failure-detection self test: one CTA waits on a shared-memory barrier that
// expects one arrival that never comes.  The bounded wait gives up after its
// wall-clock limit, records RSGPU_ERR_TIMEOUT in the error word and the kernel
// returns normally, leaving the context usable.
static __global__ void wait_for_nothing(int *err)
{
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) mbar_init(&bar, 1);
    __syncthreads();
    mbar_wait_bounded(&bar, 0, err);
}

cudaError_t launch_wait_for_nothing(int *err, cudaStream_t st)
{
    wait_for_nothing<<<1, 32, 0, st>>>(err);
    return cudaGetLastError();
}

size_t coefset_bytes(int prec) { return prec == PREC_F64 ? sizeof(CoefSet<double>) : sizeof(CoefSet<float>); }
int coef_row_stride() { return CROW; }

}  // namespace rsgpu
