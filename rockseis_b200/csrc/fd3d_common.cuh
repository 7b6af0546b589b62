// Pieces shared by the 3D propagator kernels (fd3d.cu, fd3d_elastic.cu).
#pragma once
#include "fd2d_kernels.cuh"
#include "rsgpu_3d.h"

namespace rsgpu {
namespace {

template <typename T>
__device__ __forceinline__ void load_coefs3(CoefSet3<T> &s, const CoefSet3<T> *g)
{
    const T *src = reinterpret_cast<const T *>(g);
    T *dst = reinterpret_cast<T *>(&s);
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    for (int i = tid; i < (int)(sizeof(CoefSet3<T>) / sizeof(T)); i += blockDim.x * blockDim.y) dst[i] = src[i];
}

// Staggered derivative with all NCOEF taps around b[7] (fw: b[0] = f[i-7]) or
// b[8] (bw: b[0] = f[i-8]); in both cases sum_k (b[8+k*s] - b[7-k*s]) c_k.  The
// coefficients are read from shared memory (one broadcast per tap), which keeps
// them out of the register file.
template <typename T, int MODE>
__device__ __forceinline__ T taps(const T *b, int s, const T *cu, T d, const Rcp<T> &r)
{
    using A = Ar<T, MODE>;
    T acc = A::mul(A::sub(b[8 * s], b[7 * s]), cu[0]);
#pragma unroll
    for (int k = 1; k < NCOEF; k++) acc = A::mad(acc, A::sub(b[(8 + k) * s], b[(7 - k) * s]), cu[k]);
    return (MODE == MODE_FAST) ? acc : A::div(acc, d, r);
}
template <typename T, int MODE>
__device__ __forceinline__ T taps_reg(const T (&q)[16], const T *cu, T d, const Rcp<T> &r)
{
    using A = Ar<T, MODE>;
    T acc = A::mul(A::sub(q[8], q[7]), cu[0]);
#pragma unroll
    for (int k = 1; k < NCOEF; k++) acc = A::mad(acc, A::sub(q[8 + k], q[7 - k]), cu[k]);
    return (MODE == MODE_FAST) ? acc : A::div(acc, d, r);
}

// Reduced-order form of taps_reg at a plane near an array end: K pairs (the same for the
// whole block) of the coefficient row c, the others predicated off.  The window is centred
// alike in both directions.
template <typename T, int MODE>
__device__ __forceinline__ T taps_reg_k(const T (&q)[16], int K, const T *c, T d, const Rcp<T> &r)
{
    using A = Ar<T, MODE>;
    T acc = T(0);
#pragma unroll
    for (int k = 0; k < NCOEF; k++)
        if (k < K) acc = k == 0 ? A::mul(A::sub(q[8], q[7]), c[0]) : A::mad(acc, A::sub(q[8 + k], q[7 - k]), c[k]);
    return (MODE == MODE_FAST) ? acc : A::div(acc, d, r);
}

// Two derivatives of full order on the lanes of a pair: `at(k)` the operand pair at tap k of
// the 16 (7 | 8 around the centre).
template <int MODE, typename F>
__device__ __forceinline__ float2 taps_lanes(F at, const float (&c2)[NCOEF][2], float d, const Rcp<float> &r)
{
    using A2 = Ar2<float, MODE>;
    const float2 *cc = reinterpret_cast<const float2 *>(c2);
    float2 acc = A2::mul(A2::sub(at(8), at(7)), cc[0]);
#pragma unroll
    for (int k = 1; k < NCOEF; k++) acc = A2::acc(acc, A2::sub(at(8 + k), at(7 - k)), cc[k]);
    return MODE == MODE_FAST ? acc : A2::div(acc, d, r);
}
// The same at a plane near an array end: K pairs (the same for the block) of the row c.
template <int MODE>
__device__ __forceinline__ float2 taps_lanes_k(const float2 (&q)[16], int K, const float *c, float d, const Rcp<float> &r)
{
    using A2 = Ar2<float, MODE>;
    float2 acc = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < NCOEF; k++)
        if (k < K) {
            const float2 dl = A2::sub(q[8 + k], q[7 - k]), ck = make_float2(c[k], c[k]);
            acc = k == 0 ? A2::mul(dl, ck) : A2::acc(acc, dl, ck);
        }
    return MODE == MODE_FAST ? acc : A2::div(acc, d, r);
}

// Column of the 2L strip cells of an axis that cell i holds (low strip, then high), -1: none.
__device__ __forceinline__ int strip_col(int i, int n, int L)
{
    const int c = i < L ? i : i - (n - 2 * L);
    return (i < L || i >= n - L) && i < n ? c : -1;
}
// C-PML factors A, B, C (L apart) of strip cell i; stag: at the half cells.
template <typename T>
__device__ __forceinline__ const T *strip_factors(const T *tab, int L, int i, int n, int stag)
{
    return i < L ? tab + 3 * stag * L + i : tab + (PT_RBB + 3 * stag) * L + i - (n - L);
}
// The factors of a block's columns and rows: [0] at the grid points, [1] staggered.
template <int TY>
struct PmlBlock3 {
    float x[2][3][TX3], y[2][3][TY];
};
template <int TY>
__device__ __forceinline__ void stage_pml3(PmlBlock3<TY> &p, const float *tab, int L, int x0, int y0, int nxp, int nyp)
{
    const int t = threadIdx.y * blockDim.x + threadIdx.x;
    if (t >= TX3 + TY) return;
    const bool isx = t < TX3;
    const int i = isx ? x0 + t : y0 + t - TX3, n = isx ? nxp : nyp;
    const bool in = strip_col(i, n, L) >= 0;
#pragma unroll
    for (int q = 0; q < 6; q++) {
        const float v = in ? __ldg(strip_factors(tab, L, i, n, q / 3) + q % 3 * L) : 0.f;
        if (isx) p.x[q / 3][q % 3][t] = v;
        else p.y[q / 3][q % 3][t - TX3] = v;
    }
}

// Allocation row of plane iz, padded row iy_alloc (guards included).
__device__ __forceinline__ int alloc_row3(const Shot3D<float> &sh, int iz, int iy_alloc)
{
    return (GUARD + iz) * sh.rows + iy_alloc;
}

}  // namespace
}  // namespace rsgpu
