// 2D staggered-grid finite-difference propagators for sm_100a (kernel templates).
//
// One kernel per half-step (velocity, stress), each covering every shot of a
// batch in one launch: the grid walks a table of (shot, tile) work items, so
// shots with different aperture windows share a launch.  Each CTA stages the
// stencil inputs of its TX x TZ tile, with an 8-cell halo along the axes that each is
// differentiated along, in shared memory with TMA (cp.async.bulk.tensor, completion
// on an mbarrier), while its threads fetch the point-wise inputs (velocities, moduli)
// straight into registers.  Every thread then produces a 4(x) x RZ(z) block with the
// C-PML memory-variable update and correction fused into the same pass:
//   - x-derivatives: one 128-bit shared load per 4 taps, scalar arithmetic;
//   - z-derivatives: exact, column pairs from 64-bit shared loads (dz_pair); fast, the
//     window rows streamed as 128-bit loads into paired FMAs (dz_stream_f32);
//   - the full-order coefficients are operands in the launch's parameter space; tiles
//     within `order` cells of an array end predicate off the taps that their rows and
//     columns lack (coefficient rows in shared memory).
//
// Arithmetic follows the reference operation by operation (Der::ddx_fw etc. in
// lib/der.cpp:155-540, WavesAcoustic2D/WavesElastic2D::forwardstep* in
// lib/waves.cpp:217-404, 1416-1735, backwardstep* in lib/waves.cpp:1738-2080):
//   MODE_IEEE : every add/sub/mul is a separately rounded IEEE op in the
//               reference's order, and so is the final division by the spacing: in
//               float by the two-operation formula of Rcp (rsgpu_internal.h), in
//               double where that does not serve.  Against __fdiv_rn on B200: 24 shots of
//               641 x 241, 400 steps 69 -> 43 ms, four elastic ones of 461 x 361 43 -> 23;
//   MODE_FAST : FMA contraction, coefficients pre-divided by the spacing.
#pragma once
#include <cuda.h>
#include <cstdint>
#include <type_traits>
#include "rsgpu.h"
#include "rsgpu_internal.h"
#include "rsgpu_kernels.h"
#include "exact_div.cuh"
#include "pdl.cuh"
#include "smem_limit.h"

namespace rsgpu {

enum { MODE_IEEE = 0, MODE_FAST = 2 };

// ------------------------------------------------------------------ scalar arithmetic
template <typename T, int MODE> struct Ar;
template <int MODE> struct Ar<float, MODE> {
    static constexpr bool exact = MODE != MODE_FAST;
    static __device__ __forceinline__ float add(float a, float b) { return exact ? __fadd_rn(a, b) : a + b; }
    static __device__ __forceinline__ float sub(float a, float b) { return exact ? __fsub_rn(a, b) : a - b; }
    static __device__ __forceinline__ float mul(float a, float b) { return exact ? __fmul_rn(a, b) : a * b; }
    // a + b*c (product rounded separately in the exact modes)
    static __device__ __forceinline__ float mad(float a, float b, float c)
    {
        return exact ? __fadd_rn(a, __fmul_rn(b, c)) : fmaf(b, c, a);
    }
    // a - b*c
    static __device__ __forceinline__ float msub(float a, float b, float c)
    {
        return exact ? __fsub_rn(a, __fmul_rn(b, c)) : fmaf(-b, c, a);
    }
    static __device__ __forceinline__ float div(float a, float d, const Rcp<float> &r) { return div_by(a, d, r); }
};
template <int MODE> struct Ar<double, MODE> {
    static constexpr bool exact = true;
    static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
    static __device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
    static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
    static __device__ __forceinline__ double mad(double a, double b, double c) { return __dadd_rn(a, __dmul_rn(b, c)); }
    static __device__ __forceinline__ double msub(double a, double b, double c) { return __dsub_rn(a, __dmul_rn(b, c)); }
    static __device__ __forceinline__ double div(double a, double d, const Rcp<double> &r) { return div_by(a, d, r); }
};

// ------------------------------------------------------------------ paired arithmetic (x-neighbour columns)
template <typename T> struct Pair;
template <> struct Pair<float> { using t = float2; };
template <> struct Pair<double> { using t = double2; };

template <typename T, int MODE> struct Ar2;
// Fast mode uses the paired FADD2/FMUL2/FFMA2 instructions; the exact modes
// evaluate the two lanes with separately rounded scalar operations.
template <int MODE> struct Ar2<float, MODE> {
    using P = float2;
    static constexpr bool exact = MODE != MODE_FAST;
    static __device__ __forceinline__ P mk(float a) { return make_float2(a, a); }
    static __device__ __forceinline__ P add(P a, P b)
    {
        return exact ? make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y)) : __fadd2_rn(a, b);
    }
    static __device__ __forceinline__ P sub(P a, P b)
    {
        return exact ? make_float2(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y)) : __fadd2_rn(a, make_float2(-b.x, -b.y));
    }
    static __device__ __forceinline__ P mul(P a, P b)
    {
        return exact ? make_float2(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)) : __fmul2_rn(a, b);
    }
    static __device__ __forceinline__ P acc(P s, P d, P c)
    {
        return exact ? make_float2(__fadd_rn(s.x, __fmul_rn(d.x, c.x)), __fadd_rn(s.y, __fmul_rn(d.y, c.y)))
                     : __ffma2_rn(d, c, s);
    }
    static __device__ __forceinline__ P div(P a, float d, const Rcp<float> &r)
    {
        return make_float2(div_by(a.x, d, r), div_by(a.y, d, r));
    }
};
template <int MODE> struct Ar2<double, MODE> {
    using P = double2;
    static constexpr bool exact = true;
    static __device__ __forceinline__ P mk(double a) { return make_double2(a, a); }
    static __device__ __forceinline__ P add(P a, P b) { return make_double2(__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y)); }
    static __device__ __forceinline__ P sub(P a, P b) { return make_double2(__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y)); }
    static __device__ __forceinline__ P mul(P a, P b) { return make_double2(__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)); }
    static __device__ __forceinline__ P acc(P s, P d, P c) { return add(s, mul(d, c)); }
    static __device__ __forceinline__ P div(P a, double d, const Rcp<double> &) { return make_double2(__ddiv_rn(a.x, d), __ddiv_rn(a.y, d)); }
};

template <typename T> struct Vec4;
template <> struct Vec4<float> { using type = float4; };
template <> struct Vec4<double> { using type = double4; };

template <typename T>
__device__ __forceinline__ void ld4(const T *p, T (&v)[4])
{
    typename Vec4<T>::type q = *reinterpret_cast<const typename Vec4<T>::type *>(p);
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
__device__ __forceinline__ void ldg4(const float *p, float (&v)[4])
{
    const float4 q = __ldg(reinterpret_cast<const float4 *>(p));
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
__device__ __forceinline__ void ldg4(const double *p, double (&v)[4])
{
    const double2 a = __ldg(reinterpret_cast<const double2 *>(p)), b = __ldg(reinterpret_cast<const double2 *>(p) + 1);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}

// Number of coefficient pairs the reference uses at index i of an axis of
// length n (last writer wins in lib/der.cpp's three loops).
__device__ __forceinline__ int kfw(int i, int n, int order)
{
    if (i >= n - 1) return 0;
    if (i >= n - order - 1) return n - 1 - i;
    if (i >= order - 1) return order;
    return i + 1;
}
__device__ __forceinline__ int kbw(int i, int n, int order)
{
    if (i >= n) return 0;   // padding lanes beyond the array (never stored)
    if (i >= n - order) return n - i;
    if (i >= order) return order;
    return i;   // i == 0 gives 0
}

// Coefficient rows in shared memory, row stride 9 so that a warp reading rows
// K = 0..8 touches nine distinct banks.
constexpr int CROW = 9;
template <typename T>
struct CoefSet {
    T cx[9 * CROW];   // x-direction table (pre-divided by dx in fast mode)
    T cz[9 * CROW];
};
// ------------------------------------------------------------------ TMA + mbarrier (bounded waits)
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t *bar, uint32_t phase)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(smem_u32(bar)), "r"(phase)
                 : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t global_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// Wait for the barrier phase with a wall-clock limit; on timeout record an
// error code for the host and report failure (the caller then skips its work).
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t phase, int *err)
{
    if (mbar_test(bar, phase)) return true;
    const uint64_t t0 = global_ns();
    while (!mbar_test(bar, phase)) {
        if (global_ns() - t0 > 2000000000ull) {   // 2 s
            if (err) atomicExch(err, RSGPU_ERR_TIMEOUT);
            return false;
        }
        __nanosleep(64);
    }
    return true;
}
// 2D tiled TMA load of a box at element coordinates (x, y) into shared memory.
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, uint64_t *bar, int x, int y)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}

// ------------------------------------------------------------------ derivative blocks
// x-derivative of a quad of 4 outputs on shared row `srow` (pointer at the
// quad's first halo column).  FW: f[i+k+1]-f[i-k]; BW: f[i+k]-f[i-k-1]
// (lib/der.cpp:183-188, 378-383).  `cu` = the full-order coefficients.  EDGE (tiles that
// hold reduced-order columns): output j takes its own K[j] pairs of the coefficient row
// `tab` + K[j]*CROW, taps beyond K[j] predicated off, so the lanes of a warp stay
// together: 2450 -> 1210 cycles a tile on B200 (two rows a thread, one CTA on the SM)
// against recomputing the reduced outputs one by one.
template <typename T, int MODE, bool FW, bool EDGE>
__device__ __forceinline__ void dx_quad(const T *srow, const T (&cu)[NCOEF], const T *tab, const int (&K)[4], T d,
                                        const Rcp<T> &r, T (&out)[4])
{
    using A = Ar<T, MODE>;
    T v[20];
#pragma unroll
    for (int q = 0; q < 5; q++) {
        T t[4];
        ld4(srow + 4 * q, t);
        v[4 * q] = t[0]; v[4 * q + 1] = t[1]; v[4 * q + 2] = t[2]; v[4 * q + 3] = t[3];
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        T acc = T(0);
#pragma unroll
        for (int k = 0; k < NCOEF; k++) {
            const T dl = FW ? A::sub(v[j + 9 + k], v[j + 8 - k]) : A::sub(v[j + 8 + k], v[j + 7 - k]);
            if (EDGE) {
                const T c = tab[K[j] * CROW + k];
                if (k < K[j]) acc = (k == 0) ? A::mul(dl, c) : A::mad(acc, dl, c);
            } else {
                acc = (k == 0) ? A::mul(dl, cu[k]) : A::mad(acc, dl, cu[k]);
            }
        }
        out[j] = acc;
    }
    if (MODE != MODE_FAST) div_by4(out, d, r);
}

// z-differences (before the division by the spacing) of a column pair (local columns
// c, c+1 of the tile, as one 64-bit lane pair) for RZ rows starting at tile row zr.
// Window of RZ+16 rows.
// EDGE: row rr takes its K[rr] pairs, as in dx_quad.
template <typename T, int MODE, bool FW, bool EDGE, int W, int RZ>
__device__ __forceinline__ void dz_pair(const T *s, int zr, int col, const T (&cu)[NCOEF], const T *tab,
                                        const int (&K)[RZ], typename Pair<T>::t (&out)[RZ])
{
    using A2 = Ar2<T, MODE>;
    using P = typename Pair<T>::t;
    P w[RZ + 16];
#pragma unroll
    for (int q = 0; q < RZ + 16; q++) w[q] = *reinterpret_cast<const P *>(s + (zr + q) * W + col);
#pragma unroll
    for (int rr = 0; rr < RZ; rr++) {
        P acc = A2::mk(T(0));
#pragma unroll
        for (int k = 0; k < NCOEF; k++) {
            const P dl = FW ? A2::sub(w[rr + 9 + k], w[rr + 8 - k]) : A2::sub(w[rr + 8 + k], w[rr + 7 - k]);
            if (EDGE) {
                const P c = A2::mk(tab[K[rr] * CROW + k]);
                if (k < K[rr]) acc = (k == 0) ? A2::mul(dl, c) : A2::acc(acc, dl, c);
            } else {
                const P c = A2::mk(cu[k]);
                acc = (k == 0) ? A2::mul(dl, c) : A2::acc(acc, dl, c);
            }
        }
        out[rr] = acc;
    }
}

// ------------------------------------------------------------------ C-PML helpers
__device__ __forceinline__ int xstrip(int ix, int nxp, int lpml, int &tab_base, int &col)
{
    if (ix < lpml) { tab_base = 0; col = ix; return ix; }
    const int r = ix - (nxp - lpml);
    if (r >= 0 && ix < nxp) { tab_base = 6; col = lpml + r; return r; }
    return -1;
}
__device__ __forceinline__ int zstrip(int iz, int nzp, int lpml, int &tab_base, int &row)
{
    if (iz < lpml) { tab_base = 0; row = iz; return iz; }
    const int r = iz - (nzp - lpml);
    if (r >= 0 && iz < nzp) { tab_base = 6; row = lpml + r; return r; }
    return -1;
}
// psi = B*psi + A*df ;  F -= a*(psi + C*df)   (lib/waves.cpp:252-253)
template <typename T, int MODE>
__device__ __forceinline__ T pml_correct(T F, T a, T df, T *psi, const T *tab, int lp, int base, int idx)
{
    using A = Ar<T, MODE>;
    const T tA = __ldg(tab + (base + PT_A) * lp + idx);
    const T tB = __ldg(tab + (base + PT_B) * lp + idx);
    const T tC = __ldg(tab + (base + PT_C) * lp + idx);
    T p = *psi;
    p = A::mad(A::mul(tB, p), tA, df);
    *psi = p;
    return A::msub(F, a, A::mad(p, tC, df));
}

// ------------------------------------------------------------------ tile bookkeeping
template <typename T, int TX, int TZ, int RZ>
struct Geo2D {
    static constexpr int NTX = TX / 4, NTZ = TZ / RZ, NT = NTX * NTZ;
    static constexpr int W = TX + 2 * GUARD, H = TZ + 2 * GUARD;
};

// Shared-memory prologue shared by all 2D kernels: nfield halo'd tiles (TMA),
// the coefficient tables and one mbarrier.
// HALO: per staged field the axes that carry a halo (halo_2d); a field that is
// differentiated along one axis only needs none along the other, which leaves that much
// less to fetch from L2 and more of the SM's memory to the L1 its point-wise loads pass
// through (B200, 600 steps of sixteen 861 x 461 elastic shots 77 -> 73 ms).
template <typename T, int TX, int TZ, int... HALO>
struct Smem2D {
    __host__ __device__ static constexpr int tile_bytes(int halo)
    {
        return (int)sizeof(T) * (TX + (halo & HALO_X ? 2 * GUARD : 0)) * (TZ + (halo & HALO_Z ? 2 * GUARD : 0));
    }
    __host__ __device__ static constexpr int halo(int f)
    {
        const int h[] = {HALO...};
        return h[f];
    }
    __host__ __device__ static constexpr int nfield() { return (int)sizeof...(HALO); }
    __host__ __device__ static constexpr size_t off(int f)
    {
        size_t o = 0;
        for (int k = 0; k < f; k++) o += (tile_bytes(halo(k)) + 127) / 128 * 128;
        return o;
    }
    __host__ __device__ static constexpr size_t bar_off() { return (off(nfield()) + sizeof(CoefSet<T>) + 15) / 16 * 16; }
    __host__ __device__ static constexpr size_t pml_off() { return bar_off() + 16; }
    __host__ __device__ static constexpr size_t shot_off() { return pml_off() + 6 * (TX + TZ) * sizeof(T); }
    __host__ __device__ static constexpr size_t bytes() { return shot_off() + sizeof(Shot2D<T>); }
    // field f's tile, moved so that [row + GUARD][column + GUARD] is the tile's (row, column)
    // on the axes it is differentiated along, at its own row length
    static __device__ __forceinline__ T *tile(unsigned char *sm, int f)
    {
        T *t = reinterpret_cast<T *>(sm + off(f));
        return t - (halo(f) & HALO_Z ? 0 : GUARD * (TX + 2 * GUARD)) - (halo(f) & HALO_X ? 0 : GUARD);
    }
};

template <typename T>
__device__ __forceinline__ void load_coefs(CoefSet<T> &s, const CoefSet<T> *g)
{
    const T *src = reinterpret_cast<const T *>(g);
    T *dst = reinterpret_cast<T *>(&s);
    for (int i = threadIdx.x; i < (int)(sizeof(CoefSet<T>) / sizeof(T)); i += blockDim.x) dst[i] = src[i];
}

// Copy a descriptor or table to shared memory, word by word over nt threads: one round trip
// for all of a descriptor's pointers, and the kernel's stores cannot alias it.  Visible
// after the block's next barrier.
template <typename S>
__device__ __forceinline__ void stage_words(S &dst, const S *src, int t, int nt)
{
    static_assert(sizeof(S) % sizeof(int) == 0, "whole words");
    for (int i = t; i < (int)(sizeof(S) / sizeof(int)); i += nt)
        reinterpret_cast<int *>(&dst)[i] = reinterpret_cast<const int *>(src)[i];
}

// The prologue of a tile kernel.  The first thread waits for the kernels before and issues
// the TMA loads of the fields' tiles into consecutive places; meanwhile the
// other warps bring the shot descriptor and, for edge tiles, the coefficient rows to shared
// memory.  Ends with a block barrier, after which every thread has waited.
template <typename S, typename T, int NT, int N>
__device__ __forceinline__ void tile_prologue(unsigned char *sm, uint64_t *bar, const CUtensorMap *maps,
                                              const int (&field)[N], const Tile2D &tl, Shot2D<T> &sh,
                                              const Shot2D<T> *shots, CoefSet<T> &cs, const CoefSet<T> *coefs)
{
    static_assert(N == S::nfield(), "one field a tile");
    constexpr int FIRST = NT > 32 ? 32 : 0;
    if ((int)threadIdx.x >= FIRST) {
        const int t = threadIdx.x - FIRST, nt = NT - FIRST;
        stage_words(sh, shots + tl.shot, t, nt);
        if (tl.flags & (TILE_XEDGE | TILE_ZEDGE)) stage_words(cs, coefs, t, nt);
    }
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        pdl_wait();
        uint32_t total = 0;
#pragma unroll
        for (int m = 0; m < N; m++) total += S::tile_bytes(S::halo(m));
        mbar_expect_tx(bar, total);
        // element (x0 - GUARD, z0 - GUARD) of the field is element (x0, z0) of the allocation
#pragma unroll
        for (int m = 0; m < N; m++)
            tma_load_2d(sm + S::off(m), maps + tl.shot * NMAP2D + field[m], bar, tl.x0 + (S::halo(m) & HALO_X ? 0 : GUARD),
                        tl.z0 + (S::halo(m) & HALO_Z ? 0 : GUARD));
    }
    __syncthreads();
    pdl_wait();
    pdl_trigger();
}

// ------------------------------------------------------------------ acoustic 2D
// Field tensor maps per shot: [0] P, [1] Vx, [2] Vz  (acoustic)
//                             [0] Vx, [1] Vz, [2] Sxx, [3] Szz, [4] Sxz (elastic)

// Reduced-order stencil of K pairs at one point (reference rule near the array
// ends): taps read from memory at `stride`, K known only at run time.  Two forms with
// the same operations in the same order: a call (stencil_k), for the fused 2D step and
// the plain elastic 3D kernels, where the inlined form costs the caller registers
// (-17 % there on B200); and an inlined form unrolled over the NCOEF taps with the taps
// k >= K predicated off (stencil_ki), for the 3D kernels that choose per block (TMA) and
// the plain acoustic ones (+14 %).
template <typename T, int MODE>
__device__ __noinline__ T stencil_k(const T *center, int stride, int K, const T *c, bool fw, T d, const Rcp<T> &r)
{
    using A = Ar<T, MODE>;
    if (K == 0) return T(0);
    T acc = A::mul(fw ? A::sub(center[stride], center[0]) : A::sub(center[0], center[-stride]), c[0]);
    for (int k = 1; k < K; k++) {
        const T dl = fw ? A::sub(center[(k + 1) * stride], center[-k * stride])
                        : A::sub(center[k * stride], center[-(k + 1) * stride]);
        acc = A::mad(acc, dl, c[k]);
    }
    return (MODE == MODE_FAST) ? acc : A::div(acc, d, r);
}
template <typename T, int MODE>
__device__ __forceinline__ T stencil_ki(const T *center, int stride, int K, const T *c, bool fw, T d, const Rcp<T> &r)
{
    using A = Ar<T, MODE>;
    if (K == 0) return T(0);
    T acc = A::mul(fw ? A::sub(center[stride], center[0]) : A::sub(center[0], center[-stride]), c[0]);
#pragma unroll
    for (int k = 1; k < NCOEF; k++) {
        if (k < K) {
            const T dl = fw ? A::sub(center[(k + 1) * stride], center[-k * stride])
                            : A::sub(center[k * stride], center[-(k + 1) * stride]);
            acc = A::mad(acc, dl, c[k]);
        }
    }
    return (MODE == MODE_FAST) ? acc : A::div(acc, d, r);
}
template <typename T, int MODE, int TX, int TZ, int RZ>
__device__ __forceinline__ void row_dx(const T *tile, int row, int xq, const CoefSet<T> &cs, const T (&cu)[NCOEF],
                                       bool fw, bool xedge, int gx, int nxp, int order, T d, const Rcp<T> &r, T (&out)[4])
{
    using G = Geo2D<T, TX, TZ, RZ>;
    const T *srow = tile + row * G::W + xq;
    int K[4] = {0, 0, 0, 0};
    if (xedge) {
#pragma unroll
        for (int j = 0; j < 4; j++) K[j] = fw ? kfw(gx + j, nxp, order) : kbw(gx + j, nxp, order);
        if (fw) dx_quad<T, MODE, true, true>(srow, cu, cs.cx, K, d, r, out);
        else dx_quad<T, MODE, false, true>(srow, cu, cs.cx, K, d, r, out);
    } else if (fw) {
        dx_quad<T, MODE, true, false>(srow, cu, cs.cx, K, d, r, out);
    } else {
        dx_quad<T, MODE, false, false>(srow, cu, cs.cx, K, d, r, out);
    }
}

// FAST-mode z-derivatives of the thread's 4 columns x RZ rows, streamed: each
// of the RZ+16 window rows is read once as a 128-bit shared load and scattered
// into the RZ accumulators with paired FMAs (c*w+ and -c*w- as separate terms),
// so neither the window nor a difference is held in registers.  Same taps and
// coefficients as dz_pair; only the summation order differs.  c2: every coefficient twice,
// then negated twice, in the launch's parameter space, so that a paired FMA takes it as
// a constant operand.
template <int W, int RZ, bool FW>
__device__ __forceinline__ void dz_stream_f32(const float *s, int zr, int col, const float (&c2)[2][NCOEF][2],
                                              float (&out)[RZ][4])
{
    float2 lo[RZ], hi[RZ];
#pragma unroll
    for (int rr = 0; rr < RZ; rr++) { lo[rr] = make_float2(0.f, 0.f); hi[rr] = lo[rr]; }
#pragma unroll
    for (int q = 0; q < RZ + 16; q++) {
        const float4 w = *reinterpret_cast<const float4 *>(s + (zr + q) * W + col);
        const float2 wl = make_float2(w.x, w.y), wh = make_float2(w.z, w.w);
#pragma unroll
        for (int rr = 0; rr < RZ; rr++) {
            // forward: d = sum_k c_k (w[rr+9+k] - w[rr+8-k]); backward: (w[rr+8+k] - w[rr+7-k])
            const int kp = FW ? q - rr - 9 : q - rr - 8;
            const int km = FW ? rr + 8 - q : rr + 7 - q;
            if (kp >= 0 && kp < NCOEF) {
                const float2 c = *reinterpret_cast<const float2 *>(c2[0][kp]);
                lo[rr] = __ffma2_rn(wl, c, lo[rr]);
                hi[rr] = __ffma2_rn(wh, c, hi[rr]);
            }
            if (km >= 0 && km < NCOEF) {
                const float2 c = *reinterpret_cast<const float2 *>(c2[1][km]);
                lo[rr] = __ffma2_rn(wl, c, lo[rr]);
                hi[rr] = __ffma2_rn(wh, c, hi[rr]);
            }
        }
    }
#pragma unroll
    for (int rr = 0; rr < RZ; rr++) {
        out[rr][0] = lo[rr].x; out[rr][1] = lo[rr].y; out[rr][2] = hi[rr].x; out[rr][3] = hi[rr].y;
    }
}

// One reduced-order row of four columns (fast mode; `s` at the window's first row), taps
// from shared memory so that a window is not held beside the stream's accumulators; the
// tap order is the paired form's.
template <int W, bool FW>
__device__ __forceinline__ void dz_row_edge(const float *s, const float *c, int K, float (&out)[4])
{
    using A2 = Ar2<float, MODE_FAST>;
    float2 lo = make_float2(0.f, 0.f), hi = lo;
    const float *p = s + (FW ? 9 : 8) * W, *m = s + (FW ? 8 : 7) * W;
#pragma unroll 1
    for (int k = 0; k < K; k++, p += W, m -= W) {
        const float4 a = *reinterpret_cast<const float4 *>(p), b = *reinterpret_cast<const float4 *>(m);
        const float2 ck = A2::mk(c[k]);
        const float2 dl = A2::sub(make_float2(a.x, a.y), make_float2(b.x, b.y));
        const float2 dh = A2::sub(make_float2(a.z, a.w), make_float2(b.z, b.w));
        lo = k == 0 ? A2::mul(dl, ck) : A2::acc(lo, dl, ck);
        hi = k == 0 ? A2::mul(dh, ck) : A2::acc(hi, dh, ck);
    }
    out[0] = lo.x; out[1] = lo.y; out[2] = hi.x; out[3] = hi.y;
}

// The pair form of dz over the thread's 4 columns.
template <typename T, int MODE, int W, int RZ, bool FW, bool EDGE>
__device__ __forceinline__ void dz_quads(const T *tile, int zr, int xq, const T (&cu)[NCOEF], const T *tab,
                                         const int (&K)[RZ], T (&out)[RZ][4])
{
#pragma unroll
    for (int cp = 0; cp < 2; cp++) {
        typename Pair<T>::t o[RZ];
        dz_pair<T, MODE, FW, EDGE, W, RZ>(tile, zr, xq + GUARD + 2 * cp, cu, tab, K, o);
#pragma unroll
        for (int q = 0; q < RZ; q++) { out[q][2 * cp] = o[q].x; out[q][2 * cp + 1] = o[q].y; }
    }
}

template <typename T, int MODE, int W, int RZ, bool FW>
__device__ __forceinline__ void block_dz(const T *tile, int zr, int xq, const CoefSet<T> &cs, const T (&cu)[NCOEF],
                                         const T (&c2)[2][NCOEF][2], bool zedge, int gz, int nzp, int order, T d,
                                         const Rcp<T> &r, T (&out)[RZ][4])
{
    int K[RZ];
#pragma unroll
    for (int q = 0; q < RZ; q++) K[q] = FW ? kfw(gz + q, nzp, order) : kbw(gz + q, nzp, order);
    if constexpr (MODE == MODE_FAST && std::is_same<T, float>::value) {
        dz_stream_f32<W, RZ, FW>(tile, zr, xq + GUARD, c2, out);
        if (zedge) {
#pragma unroll
            for (int q = 0; q < RZ; q++)
                if (K[q] != order)
                    dz_row_edge<W, FW>(tile + (zr + q) * W + xq + GUARD, cs.cz + K[q] * CROW, K[q], out[q]);
        }
    } else {
        if (zedge) dz_quads<T, MODE, W, RZ, FW, true>(tile, zr, xq, cu, cs.cz, K, out);
        else dz_quads<T, MODE, W, RZ, FW, false>(tile, zr, xq, cu, cs.cz, K, out);
#pragma unroll
        for (int q = 0; q < RZ; q++) div_by4(out[q], d, r);
    }
}

// Point-wise blocks.  Rows and columns beyond the padded grid (up to the tile
// edge) lie inside the allocation; their parameters are zero, so the update
// leaves the fields there exactly zero, and loads and stores need no bounds
// checks.  `o0` is the element offset of the thread's first output.
template <typename T, int RZ>
__device__ __forceinline__ void load_block(const T *base, int o0, int pitch, T (&v)[RZ][4])
{
#pragma unroll
    for (int q = 0; q < RZ; q++) ldg4(base + o0 + q * pitch, v[q]);
}
template <typename T, int RZ>
__device__ __forceinline__ void load_block_rw(const T *base, int o0, int pitch, T (&v)[RZ][4])
{
#pragma unroll
    for (int q = 0; q < RZ; q++) ld4(base + o0 + q * pitch, v[q]);
}
template <typename T, int RZ>
__device__ __forceinline__ void store_block(T *base, int o0, int pitch, const T (&v)[RZ][4])
{
#pragma unroll
    for (int q = 0; q < RZ; q++)
        *reinterpret_cast<typename Vec4<T>::type *>(base + o0 + q * pitch) = {v[q][0], v[q][1], v[q][2], v[q][3]};
}

// ------------------------------------------------------------------ C-PML of a tile
// A tile in the strips costs its CTA latency, not bandwidth, and sets the time of a
// launch of few tiles, so: the factors A, B, C of the tile's columns and rows are
// fetched in the prologue (registers, then shared memory once the TMA wait is over), a
// thread's memory variables are all loaded before any is stored (a load that follows a
// store to memory the compiler cannot tell apart waits behind it), and the update runs
// unconditionally on zeros outside the strips with one select per point instead of a
// branch.  On B200 (fast mode) the x part of a strip tile's update went from 1910 to 170
// cycles, and with the reduced-order rows of dx_quad and dz_row_edge 600 steps of sixteen
// 861 x 461 elastic shots from 96 to 77 ms, 2000 steps of one 541 x 341 acoustic shot
// from 37 to 31.
template <typename T, int TX, int TZ>
struct PmlTile {
    T x[2][3][TX], z[2][3][TZ];   // [0] at the grid points, [1] staggered; A, B, C; zero outside the strips
};
template <typename T, int TX, int TZ, int NT>
struct PmlFetch {
    static constexpr int N = (TX + TZ + NT - 1) / NT;
    T v[N][6];
    __device__ __forceinline__ void fetch(const Step2DArgs<T> &a, const Shot2D<T> &sh, const Tile2D &tl)
    {
#pragma unroll
        for (int n = 0; n < N; n++) {
            const int t = threadIdx.x + n * NT;
            int base = 0, col = 0;
            const int i = t < TX ? xstrip(tl.x0 + t, sh.nxp, a.lpml, base, col)
                                 : t < TX + TZ ? zstrip(tl.z0 + t - TX, sh.nzp, a.lpml, base, col) : -1;
#pragma unroll
            for (int q = 0; q < 6; q++) v[n][q] = i >= 0 ? __ldg(a.pml + (base + q) * a.lpml + i) : T(0);
        }
    }
    __device__ __forceinline__ void store(PmlTile<T, TX, TZ> &p) const
    {
#pragma unroll
        for (int n = 0; n < N; n++) {
            const int t = threadIdx.x + n * NT;
#pragma unroll
            for (int q = 0; q < 6; q++) {
                if (t < TX) p.x[q / 3][q % 3][t] = v[n][q];
                else if (t < TX + TZ) p.z[q / 3][q % 3][t - TX] = v[n][q];
            }
        }
    }
};
static_assert(PT_LTF_STAG == PT_LTF + 3 && PT_RBB_STAG == PT_RBB + 3, "a staggered table follows its unstaggered one");

// A thread's memory variables of one x strip and one z strip update: a vector a row and
// strip.  in[j], zin[q]: column j in an x strip, row q in a z strip.
template <typename T, int RZ>
struct PsiBlock {
    T px[RZ][4], pz[RZ][4];
    template <bool X, bool Z>
    __device__ __forceinline__ void load(const Shot2D<T> &sh, int lpml, int flags, int gx, int gz, const T *psix,
                                         const T *psiz)
    {
        if (X && (flags & TILE_XPML)) {
            const bool quad = xquad(sh, lpml, gx);
            const T *p = psix + gz * psix_pitch(sh.nxp, lpml) + psix_col(gx, sh.nxp, lpml);
#pragma unroll
            for (int q = 0; q < RZ; q++) get(p + q * psix_pitch(sh.nxp, lpml), quad && gz + q < sh.nzp, px[q]);
        }
        if (Z && (flags & TILE_ZPML)) {
#pragma unroll
            for (int q = 0; q < RZ; q++)
                get(psiz + zrow(sh, lpml, gz + q) * psiz_pitch(sh.nxp) + gx, zin(sh, lpml, gz + q) && gx < sh.nxp, pz[q]);
        }
    }
    template <bool X, bool Z>
    __device__ __forceinline__ void store(const Shot2D<T> &sh, int lpml, int flags, int gx, int gz, T *psix,
                                          T *psiz) const
    {
        if (X && (flags & TILE_XPML)) {
            const bool quad = xquad(sh, lpml, gx);
            T *p = psix + gz * psix_pitch(sh.nxp, lpml) + psix_col(gx, sh.nxp, lpml);
#pragma unroll
            for (int q = 0; q < RZ; q++) put(p + q * psix_pitch(sh.nxp, lpml), quad && gz + q < sh.nzp, px[q]);
        }
        if (Z && (flags & TILE_ZPML)) {
#pragma unroll
            for (int q = 0; q < RZ; q++)
                put(psiz + zrow(sh, lpml, gz + q) * psiz_pitch(sh.nxp) + gx, zin(sh, lpml, gz + q) && gx < sh.nxp, pz[q]);
        }
    }
    static __device__ __forceinline__ bool xin(const Shot2D<T> &sh, int lpml, int ix)
    {
        return ix < lpml || ix >= sh.nxp - lpml;
    }
    static __device__ __forceinline__ bool zin(const Shot2D<T> &sh, int lpml, int iz)
    {
        return iz < lpml || (iz >= sh.nzp - lpml && iz < sh.nzp);
    }

private:
    static __device__ __forceinline__ bool xquad(const Shot2D<T> &sh, int lpml, int gx)
    {
        return gx < psi_left(lpml) || (gx >= psi_right(sh.nxp, lpml) && gx < sh.nxp);
    }
    static __device__ __forceinline__ int zrow(const Shot2D<T> &sh, int lpml, int iz)
    {
        return iz < lpml ? iz : iz - (sh.nzp - 2 * lpml);
    }
    static __device__ __forceinline__ void get(const T *p, bool in, T (&v)[4])
    {
        v[0] = v[1] = v[2] = v[3] = T(0);
        if (in) ld4(p, v);
    }
    static __device__ __forceinline__ void put(T *p, bool in, const T (&v)[4])
    {
        if (in) *reinterpret_cast<typename Vec4<T>::type *>(p) = {v[0], v[1], v[2], v[3]};
    }
};

// psi = B*psi + A*df and the corrected derivative term psi + C*df (lib/waves.cpp:252-253)
template <typename T, int MODE>
__device__ __forceinline__ T pml_term(T &psi, T df, T tA, T tB, T tC)
{
    using A = Ar<T, MODE>;
    psi = A::mad(A::mul(tB, psi), tA, df);
    return A::mad(psi, tC, df);
}

// x-part then z-part of one field, a = dt*modulus (lib/waves.cpp:245-307):
//   F += a*d1 ; [x strip] psi = B*psi + A*d1, F -= a*(psi + C*d1) ;
//   F += a*d2 ; [z strip] the same with the z memory variable.
// X, Z: the parts present; sx, sz: the staggered factors (1) or not (0).
template <typename T, int MODE, int TX, int TZ, int RZ, bool X, bool Z>
__device__ __forceinline__ void update_field(T (&F)[RZ][4], const T (&Mo)[RZ][4], const T (&d1)[RZ][4],
                                             const T (&d2)[RZ][4], PsiBlock<T, RZ> &ps, const PmlTile<T, TX, TZ> &pt,
                                             int sx, int sz, int flags, int gx, int gz, int xq, int zr,
                                             const Shot2D<T> &sh, const Step2DArgs<T> &a, bool const_mod)
{
    using A = Ar<T, MODE>;
#pragma unroll
    for (int part = 0; part < 2; part++) {
        if (part == 0 ? !X : !Z) continue;
        const T (&d)[RZ][4] = part == 0 ? d1 : d2;
#pragma unroll
        for (int q = 0; q < RZ; q++)
#pragma unroll
            for (int j = 0; j < 4; j++) F[q][j] = A::mad(F[q][j], const_mod ? a.dt : A::mul(a.dt, Mo[q][j]), d[q][j]);
        if (!(flags & (part == 0 ? TILE_XPML : TILE_ZPML))) continue;
        T fx[3][4];
        if (part == 0)
#pragma unroll
            for (int t = 0; t < 3; t++) ld4(pt.x[sx][t] + xq, fx[t]);
#pragma unroll
        for (int q = 0; q < RZ; q++) {
            T fz[3];
            if (part == 1)
#pragma unroll
                for (int t = 0; t < 3; t++) fz[t] = pt.z[sz][t][zr + q];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const bool in = part == 0 ? PsiBlock<T, RZ>::xin(sh, a.lpml, gx + j)
                                          : PsiBlock<T, RZ>::zin(sh, a.lpml, gz + q);
                T &p = part == 0 ? ps.px[q][j] : ps.pz[q][j];
                const T am = const_mod ? a.dt : A::mul(a.dt, Mo[q][j]);
                const T c = part == 0 ? pml_term<T, MODE>(p, d[q][j], fx[0][j], fx[1][j], fx[2][j])
                                      : pml_term<T, MODE>(p, d[q][j], fz[0], fz[1], fz[2]);
                const T G = A::msub(F[q][j], am, c);
                F[q][j] = in ? G : F[q][j];
            }
        }
    }
}

#define RS_TILE_SETUP()                                                                        \
    using G = Geo2D<T, TX, TZ, RZ>;                                                            \
    const int tx = threadIdx.x % G::NTX, tz = threadIdx.x / G::NTX;                            \
    const int xq = 4 * tx, zr = tz * RZ, gx = tl.x0 + xq, gz = tl.z0 + zr;                     \
    const int o0 = gz * sh.pitch + gx, pitch = sh.pitch, fl = tl.flags;                        \
    const bool xe = fl & TILE_XEDGE, ze = fl & TILE_ZEDGE;                                     \
    const bool pml = fl & (TILE_XPML | TILE_ZPML)

// Wait for the staged tiles (bar, null: already waited for) and, in C-PML tiles, share
// the factors; false if the wait gave up.
template <typename T, int TX, int TZ, int NT>
__device__ __forceinline__ bool tile_ready(uint64_t *bar, int *err, bool pml, const PmlFetch<T, TX, TZ, NT> &pf,
                                           PmlTile<T, TX, TZ> &pt)
{
    const bool ok = !bar || mbar_wait_bounded(bar, 0, err);
    if (!pml) return ok;
    pf.store(pt);
    return __syncthreads_and(ok);
}

// Velocity half-step: Vx += dt*Rx*Dx+P (+ x C-PML), Vz += dt*Rz*Dz+P (+ z C-PML)
// (lib/waves.cpp:217-310).
template <typename T, int MODE, int TX, int TZ, int RZ>
__device__ __forceinline__ void a2d_velocity_tile(const Step2DArgs<T> &a, const Shot2D<T> &sh, const Tile2D &tl,
                                                  const T *sP, const CoefSet<T> &cs, PmlTile<T, TX, TZ> &pt, int *err,
                                                  uint64_t *bar)
{
    RS_TILE_SETUP();
    PmlFetch<T, TX, TZ, G::NT> pf;
    PsiBlock<T, RZ> ps;
    T F[RZ][4], M[RZ][4], F2[RZ][4], M2[RZ][4], d[RZ][4];
    load_block_rw<T, RZ>(sh.f[A2_VX], o0, pitch, F);
    load_block<T, RZ>(sh.m[M_RX], o0, pitch, M);
    load_block_rw<T, RZ>(sh.f[A2_VZ], o0, pitch, F2);
    load_block<T, RZ>(sh.m[M_RZ], o0, pitch, M2);
    if (pml) {
        pf.fetch(a, sh, tl);
        ps.template load<true, true>(sh, a.lpml, fl, gx, gz, sh.psix[0], sh.psiz[0]);
    }
    if (!tile_ready(bar, err, pml, pf, pt)) return;
#pragma unroll
    for (int q = 0; q < RZ; q++) row_dx<T, MODE, TX, TZ, RZ>(sP, zr + q + GUARD, xq, cs, a.cx, true, xe, gx, sh.nxp, a.order, a.dx, a.rdx, d[q]);
    update_field<T, MODE, TX, TZ, RZ, true, false>(F, M, d, d, ps, pt, 1, 1, fl, gx, gz, xq, zr, sh, a, false);
    store_block<T, RZ>(sh.f[A2_VX], o0, pitch, F);
    block_dz<T, MODE, G::W, RZ, true>(sP, zr, xq, cs, a.cz, a.cz2, ze, gz, sh.nzp, a.order, a.dz, a.rdz, d);
    update_field<T, MODE, TX, TZ, RZ, false, true>(F2, M2, d, d, ps, pt, 1, 1, fl, gx, gz, xq, zr, sh, a, false);
    store_block<T, RZ>(sh.f[A2_VZ], o0, pitch, F2);
    if (pml) ps.template store<true, true>(sh, a.lpml, fl, gx, gz, sh.psix[0], sh.psiz[0]);
}

// Stress half-step: P += dt*L*Dx-Vx (+x C-PML), then P += dt*L*Dz-Vz (+z C-PML)
// (lib/waves.cpp:313-404).
template <typename T, int MODE, int TX, int TZ, int RZ>
__device__ __forceinline__ void a2d_stress_tile(const Step2DArgs<T> &a, const Shot2D<T> &sh, const Tile2D &tl,
                                                const T *sVx, const T *sVz, const CoefSet<T> &cs,
                                                PmlTile<T, TX, TZ> &pt, int *err, uint64_t *bar)
{
    RS_TILE_SETUP();
    PmlFetch<T, TX, TZ, G::NT> pf;
    PsiBlock<T, RZ> ps;
    T F[RZ][4], M[RZ][4], d1[RZ][4], d2[RZ][4];
    load_block_rw<T, RZ>(sh.f[A2_P], o0, pitch, F);
    load_block<T, RZ>(sh.m[M_L], o0, pitch, M);
    if (pml) {
        pf.fetch(a, sh, tl);
        ps.template load<true, true>(sh, a.lpml, fl, gx, gz, sh.psix[1], sh.psiz[1]);
    }
    if (!tile_ready(bar, err, pml, pf, pt)) return;
#pragma unroll
    for (int q = 0; q < RZ; q++) row_dx<T, MODE, TX, TZ, RZ>(sVx, zr + q + GUARD, xq, cs, a.cx, false, xe, gx, sh.nxp, a.order, a.dx, a.rdx, d1[q]);
    block_dz<T, MODE, TX, RZ, false>(sVz, zr, xq, cs, a.cz, a.cz2, ze, gz, sh.nzp, a.order, a.dz, a.rdz, d2);
    update_field<T, MODE, TX, TZ, RZ, true, true>(F, M, d1, d2, ps, pt, 0, 0, fl, gx, gz, xq, zr, sh, a, false);
    store_block<T, RZ>(sh.f[A2_P], o0, pitch, F);
    if (pml) ps.template store<true, true>(sh, a.lpml, fl, gx, gz, sh.psix[1], sh.psiz[1]);
}

// ---------------------------------------------------------------- elastic 2D
// Velocity half-step.  Forward (lib/waves.cpp:1416-1566):
//   Vx += dt*Rx*Dx+Sxx [x stag psi0] ; Vx += dt*Rx*Dz-Sxz [z psi0]
//   Vz += dt*Rz*Dx-Sxz [x psi1]      ; Vz += dt*Rz*Dz+Szz [z stag psi1]
// Adjoint (lib/waves.cpp:1738-1913): Sxx -> L2M*Sxx + L*Szz, Sxz -> M*Sxz,
// Szz -> L*Sxx + L2M*Szz (formed in shared memory after the TMA loads).
// WZZ: row length of the Szz tile (no x halo in the forward step)
template <typename T, int MODE, int TX, int TZ, int RZ, int WZZ>
__device__ __forceinline__ void e2d_velocity_tile(const Step2DArgs<T> &a, const Shot2D<T> &sh, const Tile2D &tl,
                                                  const T *sXX, const T *sZZ, const T *sXZ, const CoefSet<T> &cs,
                                                  PmlTile<T, TX, TZ> &pt, uint64_t *bar, int *err)
{
    RS_TILE_SETUP();
    PmlFetch<T, TX, TZ, G::NT> pf;
    PsiBlock<T, RZ> ps;
    T F[RZ][4], M[RZ][4], F2[RZ][4], M2[RZ][4], d1[RZ][4], d2[RZ][4];
    // all point-wise inputs of both passes are requested before the first wait
    load_block_rw<T, RZ>(sh.f[E2_VX], o0, pitch, F);
    load_block<T, RZ>(sh.m[M_RX], o0, pitch, M);
    load_block_rw<T, RZ>(sh.f[E2_VZ], o0, pitch, F2);
    load_block<T, RZ>(sh.m[M_RZ], o0, pitch, M2);
    if (pml) pf.fetch(a, sh, tl);
    if (!tile_ready(bar, err, pml, pf, pt)) return;
    if (pml) ps.template load<true, true>(sh, a.lpml, fl, gx, gz, sh.psix[0], sh.psiz[0]);
#pragma unroll
    for (int q = 0; q < RZ; q++) row_dx<T, MODE, TX, TZ, RZ>(sXX, zr + q + GUARD, xq, cs, a.cx, true, xe, gx, sh.nxp, a.order, a.dx, a.rdx, d1[q]);
    block_dz<T, MODE, G::W, RZ, false>(sXZ, zr, xq, cs, a.cz, a.cz2, ze, gz, sh.nzp, a.order, a.dz, a.rdz, d2);
    update_field<T, MODE, TX, TZ, RZ, true, true>(F, M, d1, d2, ps, pt, 1, 0, fl, gx, gz, xq, zr, sh, a, false);
    PsiBlock<T, RZ> p2;
    if (pml) p2.template load<true, true>(sh, a.lpml, fl, gx, gz, sh.psix[1], sh.psiz[1]);
    store_block<T, RZ>(sh.f[E2_VX], o0, pitch, F);
    if (pml) ps.template store<true, true>(sh, a.lpml, fl, gx, gz, sh.psix[0], sh.psiz[0]);
#pragma unroll
    for (int q = 0; q < RZ; q++) row_dx<T, MODE, TX, TZ, RZ>(sXZ, zr + q + GUARD, xq, cs, a.cx, false, xe, gx, sh.nxp, a.order, a.dx, a.rdx, d1[q]);
    block_dz<T, MODE, WZZ, RZ, true>(sZZ, zr, xq, cs, a.cz, a.cz2, ze, gz, sh.nzp, a.order, a.dz, a.rdz, d2);
    update_field<T, MODE, TX, TZ, RZ, true, true>(F2, M2, d1, d2, p2, pt, 0, 1, fl, gx, gz, xq, zr, sh, a, false);
    store_block<T, RZ>(sh.f[E2_VZ], o0, pitch, F2);
    if (pml) p2.template store<true, true>(sh, a.lpml, fl, gx, gz, sh.psix[1], sh.psiz[1]);
}

// Normal stresses of the elastic stress half-step (lib/waves.cpp:1596-1674):
//   d1 = Dx-Vx: Sxx += dt*L2M*d1, Szz += dt*L*d1, one x memory update for both;
//   d2 = Dz-Vz: Sxx += dt*L*d2,   Szz += dt*L2M*d2, one z memory update;
//   free surface: Szz = 0 on row lpml.
// Adjoint (lib/waves.cpp:1939-2018): Sxx += dt*d1, Szz += dt*d2 with their own memories.
template <typename T, int MODE, int TX, int TZ, int RZ, bool ADJ>
__device__ __forceinline__ void update_normal(T (&sxx)[RZ][4], T (&szz)[RZ][4], const T (&l)[RZ][4],
                                              const T (&l2m)[RZ][4], const T (&d1)[RZ][4], const T (&d2)[RZ][4],
                                              PsiBlock<T, RZ> &ps, const PmlTile<T, TX, TZ> &pt, int flags, int gx,
                                              int gz, int xq, int zr, const Shot2D<T> &sh, const Step2DArgs<T> &a)
{
    using A = Ar<T, MODE>;
#pragma unroll
    for (int part = 0; part < 2; part++) {
        const T (&d)[RZ][4] = part == 0 ? d1 : d2;
#pragma unroll
        for (int q = 0; q < RZ; q++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const T a2 = ADJ ? a.dt : A::mul(a.dt, l2m[q][j]), a1 = ADJ ? a.dt : A::mul(a.dt, l[q][j]);
                if (!ADJ || part == 0) sxx[q][j] = A::mad(sxx[q][j], part == 0 ? a2 : a1, d[q][j]);
                if (!ADJ || part == 1) szz[q][j] = A::mad(szz[q][j], part == 0 ? a1 : a2, d[q][j]);
            }
        if (!(flags & (part == 0 ? TILE_XPML : TILE_ZPML))) continue;
        T fx[3][4];
        if (part == 0)
#pragma unroll
            for (int t = 0; t < 3; t++) ld4(pt.x[0][t] + xq, fx[t]);
#pragma unroll
        for (int q = 0; q < RZ; q++) {
            T fz[3];
            if (part == 1)
#pragma unroll
                for (int t = 0; t < 3; t++) fz[t] = pt.z[0][t][zr + q];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const bool in = part == 0 ? PsiBlock<T, RZ>::xin(sh, a.lpml, gx + j)
                                          : PsiBlock<T, RZ>::zin(sh, a.lpml, gz + q);
                T &p = part == 0 ? ps.px[q][j] : ps.pz[q][j];
                const T a2 = ADJ ? a.dt : A::mul(a.dt, l2m[q][j]), a1 = ADJ ? a.dt : A::mul(a.dt, l[q][j]);
                const T c = part == 0 ? pml_term<T, MODE>(p, d[q][j], fx[0][j], fx[1][j], fx[2][j])
                                      : pml_term<T, MODE>(p, d[q][j], fz[0], fz[1], fz[2]);
                if (!ADJ || part == 0) {
                    const T G = A::msub(sxx[q][j], part == 0 ? a2 : a1, c);
                    sxx[q][j] = in ? G : sxx[q][j];
                }
                if (!ADJ || part == 1) {
                    const T G = A::msub(szz[q][j], part == 0 ? a1 : a2, c);
                    szz[q][j] = in ? G : szz[q][j];
                }
            }
        }
    }
#pragma unroll
    for (int q = 0; q < RZ; q++)
        if (sh.fs && gz + q == a.lpml) szz[q][0] = szz[q][1] = szz[q][2] = szz[q][3] = T(0);
}

// Stress half-step.  Forward (lib/waves.cpp:1571-1735): normal stresses as
// above, then Sxz += dt*M*Dx+Vz [x stag psi3] ; Sxz += dt*M*Dz+Vx [z stag psi3].
// Adjoint (lib/waves.cpp:1916-2080): Sxz without the modulus.
template <typename T, int MODE, int TX, int TZ, int RZ, bool ADJ>
__device__ __forceinline__ void e2d_stress_tile(const Step2DArgs<T> &a, const Shot2D<T> &sh, const Tile2D &tl,
                                                const T *sVx, const T *sVz, const CoefSet<T> &cs,
                                                PmlTile<T, TX, TZ> &pt, uint64_t *bar, int *err)
{
    RS_TILE_SETUP();
    T d1[RZ][4], d2[RZ][4], sxx[RZ][4], szz[RZ][4];
    PsiBlock<T, RZ> ps;
    {
        PmlFetch<T, TX, TZ, G::NT> pf;
        T l[RZ][4], l2m[RZ][4];
        load_block_rw<T, RZ>(sh.f[E2_SXX], o0, pitch, sxx);
        load_block_rw<T, RZ>(sh.f[E2_SZZ], o0, pitch, szz);
        if (!ADJ) {
            load_block<T, RZ>(sh.m[M_L], o0, pitch, l);
            load_block<T, RZ>(sh.m[M_L2M], o0, pitch, l2m);
        }
        // warm the shear-stress inputs of the second pass into L1/L2 meanwhile
#pragma unroll
        for (int q = 0; q < RZ; q++) {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(sh.f[E2_SXZ] + o0 + q * pitch));
            if (!ADJ) asm volatile("prefetch.global.L2 [%0];" ::"l"(sh.m[M_M] + o0 + q * pitch));
        }
        if (pml) pf.fetch(a, sh, tl);
        if (!tile_ready(bar, err, pml, pf, pt)) return;
        if (pml) ps.template load<true, true>(sh, a.lpml, fl, gx, gz, sh.psix[2], sh.psiz[2]);
#pragma unroll
        for (int q = 0; q < RZ; q++) row_dx<T, MODE, TX, TZ, RZ>(sVx, zr + q + GUARD, xq, cs, a.cx, false, xe, gx, sh.nxp, a.order, a.dx, a.rdx, d1[q]);
        block_dz<T, MODE, G::W, RZ, false>(sVz, zr, xq, cs, a.cz, a.cz2, ze, gz, sh.nzp, a.order, a.dz, a.rdz, d2);
        update_normal<T, MODE, TX, TZ, RZ, ADJ>(sxx, szz, l, l2m, d1, d2, ps, pt, fl, gx, gz, xq, zr, sh, a);
    }
    {
        // the shear inputs are requested before the normal stresses are stored: a
        // load that follows a store to memory the compiler cannot tell apart waits
        // behind it
        T F[RZ][4], M[RZ][4];
        PsiBlock<T, RZ> p2;
        load_block_rw<T, RZ>(sh.f[E2_SXZ], o0, pitch, F);
        if (!ADJ) load_block<T, RZ>(sh.m[M_M], o0, pitch, M);
        if (pml) p2.template load<true, true>(sh, a.lpml, fl, gx, gz, sh.psix[3], sh.psiz[3]);
        store_block<T, RZ>(sh.f[E2_SXX], o0, pitch, sxx);
        store_block<T, RZ>(sh.f[E2_SZZ], o0, pitch, szz);
        if (pml) ps.template store<true, true>(sh, a.lpml, fl, gx, gz, sh.psix[2], sh.psiz[2]);
#pragma unroll
        for (int q = 0; q < RZ; q++) row_dx<T, MODE, TX, TZ, RZ>(sVz, zr + q + GUARD, xq, cs, a.cx, true, xe, gx, sh.nxp, a.order, a.dx, a.rdx, d1[q]);
        block_dz<T, MODE, G::W, RZ, true>(sVx, zr, xq, cs, a.cz, a.cz2, ze, gz, sh.nzp, a.order, a.dz, a.rdz, d2);
        update_field<T, MODE, TX, TZ, RZ, true, true>(F, M, d1, d2, p2, pt, 1, 1, fl, gx, gz, xq, zr, sh, a, ADJ);
        store_block<T, RZ>(sh.f[E2_SXZ], o0, pitch, F);
        if (pml) p2.template store<true, true>(sh, a.lpml, fl, gx, gz, sh.psix[3], sh.psiz[3]);
    }
}

// ------------------------------------------------------------------ kernels
template <typename T, int TX, int TZ> using SmemA2V = Smem2D<T, TX, TZ, halo_2d(PHYS_A2D, A2_P, false)>;
template <typename T, int TX, int TZ>
using SmemA2S = Smem2D<T, TX, TZ, halo_2d(PHYS_A2D, A2_VX, false), halo_2d(PHYS_A2D, A2_VZ, false)>;
template <typename T, int TX, int TZ, bool ADJ>
using SmemE2V = Smem2D<T, TX, TZ, halo_2d(PHYS_E2D, E2_SXX, ADJ), halo_2d(PHYS_E2D, E2_SZZ, ADJ), halo_2d(PHYS_E2D, E2_SXZ, ADJ)>;
template <typename T, int TX, int TZ>
using SmemE2S = Smem2D<T, TX, TZ, halo_2d(PHYS_E2D, E2_VX, false), halo_2d(PHYS_E2D, E2_VZ, false)>;

template <typename T, int MODE, int TX, int TZ, int RZ, int MINB>
__global__ void __launch_bounds__(Geo2D<T, TX, TZ, RZ>::NT, MINB)
a2d_velocity(Step2DArgs<T> a, const CoefSet<T> *coefs, const CUtensorMap *maps, int *err)
{
    using G = Geo2D<T, TX, TZ, RZ>;
    using S = SmemA2V<T, TX, TZ>;
    extern __shared__ __align__(128) unsigned char sm[];
    CoefSet<T> &cs = *reinterpret_cast<CoefSet<T> *>(sm + S::off(S::nfield()));
    uint64_t *bar = reinterpret_cast<uint64_t *>(sm + S::bar_off());
    PmlTile<T, TX, TZ> &pt = *reinterpret_cast<PmlTile<T, TX, TZ> *>(sm + S::pml_off());
    Shot2D<T> &sh = *reinterpret_cast<Shot2D<T> *>(sm + S::shot_off());
    const Tile2D tl = a.tiles[blockIdx.x];
    const int field[] = {A2_P};
    tile_prologue<S, T, G::NT>(sm, bar, maps, field, tl, sh, a.shots, cs, coefs);
    const T *sP = S::tile(sm, 0);
    a2d_velocity_tile<T, MODE, TX, TZ, RZ>(a, sh, tl, sP, cs, pt, err, bar);
}

template <typename T, int MODE, int TX, int TZ, int RZ, int MINB>
__global__ void __launch_bounds__(Geo2D<T, TX, TZ, RZ>::NT, MINB)
a2d_stress(Step2DArgs<T> a, const CoefSet<T> *coefs, const CUtensorMap *maps, int *err)
{
    using G = Geo2D<T, TX, TZ, RZ>;
    using S = SmemA2S<T, TX, TZ>;
    extern __shared__ __align__(128) unsigned char sm[];
    CoefSet<T> &cs = *reinterpret_cast<CoefSet<T> *>(sm + S::off(S::nfield()));
    uint64_t *bar = reinterpret_cast<uint64_t *>(sm + S::bar_off());
    PmlTile<T, TX, TZ> &pt = *reinterpret_cast<PmlTile<T, TX, TZ> *>(sm + S::pml_off());
    Shot2D<T> &sh = *reinterpret_cast<Shot2D<T> *>(sm + S::shot_off());
    const Tile2D tl = a.tiles[blockIdx.x];
    const int field[] = {A2_VX, A2_VZ};
    tile_prologue<S, T, G::NT>(sm, bar, maps, field, tl, sh, a.shots, cs, coefs);
    const T *sVx = S::tile(sm, 0), *sVz = S::tile(sm, 1);
    a2d_stress_tile<T, MODE, TX, TZ, RZ>(a, sh, tl, sVx, sVz, cs, pt, err, bar);
}

// Adjoint work arrays in place: wrk1 = L2M*Sxx + L*Szz, wrk3 = L*Sxx + L2M*Szz,
// wrk2 = M*Sxz (lib/waves.cpp:1774, 1812, 1885), over the whole halo'd tile.
template <typename T, int MODE, int TX, int TZ, int RZ>
__device__ __forceinline__ void adjoint_work(T *sXX, T *sZZ, T *sXZ, const Shot2D<T> &sh, int x0, int z0)
{
    using G = Geo2D<T, TX, TZ, RZ>;
    using A = Ar<T, MODE>;
    const long off0 = (long)(z0 - GUARD) * sh.pitch + (x0 - GUARD);
    for (int q = threadIdx.x; q < G::W * G::H; q += G::NT) {
        const int rr = q / G::W, c = q - rr * G::W;
        const long o = off0 + (long)rr * sh.pitch + c;
        const T sxx = sXX[q], szz = sZZ[q], l = sh.m[M_L][o], l2m = sh.m[M_L2M][o], m = sh.m[M_M][o];
        sXX[q] = A::add(A::mul(l2m, sxx), A::mul(l, szz));
        sZZ[q] = A::add(A::mul(l, sxx), A::mul(l2m, szz));
        sXZ[q] = A::mul(m, sXZ[q]);
    }
}

template <typename T, int MODE, int TX, int TZ, int RZ, int MINB, bool ADJ>
__global__ void __launch_bounds__(Geo2D<T, TX, TZ, RZ>::NT, MINB)
e2d_velocity(Step2DArgs<T> a, const CoefSet<T> *coefs, const CUtensorMap *maps, int *err)
{
    using G = Geo2D<T, TX, TZ, RZ>;
    using S = SmemE2V<T, TX, TZ, ADJ>;
    extern __shared__ __align__(128) unsigned char sm[];
    CoefSet<T> &cs = *reinterpret_cast<CoefSet<T> *>(sm + S::off(S::nfield()));
    uint64_t *bar = reinterpret_cast<uint64_t *>(sm + S::bar_off());
    PmlTile<T, TX, TZ> &pt = *reinterpret_cast<PmlTile<T, TX, TZ> *>(sm + S::pml_off());
    Shot2D<T> &sh = *reinterpret_cast<Shot2D<T> *>(sm + S::shot_off());
    const Tile2D tl = a.tiles[blockIdx.x];
    const int field[] = {E2_SXX, E2_SZZ, E2_SXZ};
    tile_prologue<S, T, G::NT>(sm, bar, maps, field, tl, sh, a.shots, cs, coefs);
    T *sXX = S::tile(sm, 0), *sZZ = S::tile(sm, 1),
      *sXZ = S::tile(sm, 2);
    uint64_t *wbar = bar;
    if (ADJ) {
        // every thread reaches the same barriers whether or not the wait succeeded
        const bool ok = __syncthreads_and(mbar_wait_bounded(bar, 0, err));
        if (!ok) return;
        adjoint_work<T, MODE, TX, TZ, RZ>(sXX, sZZ, sXZ, sh, tl.x0, tl.z0);
        __syncthreads();
        wbar = nullptr;
    }
    e2d_velocity_tile<T, MODE, TX, TZ, RZ, ADJ ? G::W : TX>(a, sh, tl, sXX, sZZ, sXZ, cs, pt, wbar, err);
}

template <typename T, int MODE, int TX, int TZ, int RZ, int MINB, bool ADJ>
__global__ void __launch_bounds__(Geo2D<T, TX, TZ, RZ>::NT, MINB)
e2d_stress(Step2DArgs<T> a, const CoefSet<T> *coefs, const CUtensorMap *maps, int *err)
{
    using G = Geo2D<T, TX, TZ, RZ>;
    using S = SmemE2S<T, TX, TZ>;
    extern __shared__ __align__(128) unsigned char sm[];
    CoefSet<T> &cs = *reinterpret_cast<CoefSet<T> *>(sm + S::off(S::nfield()));
    uint64_t *bar = reinterpret_cast<uint64_t *>(sm + S::bar_off());
    PmlTile<T, TX, TZ> &pt = *reinterpret_cast<PmlTile<T, TX, TZ> *>(sm + S::pml_off());
    Shot2D<T> &sh = *reinterpret_cast<Shot2D<T> *>(sm + S::shot_off());
    const Tile2D tl = a.tiles[blockIdx.x];
    const int field[] = {E2_VX, E2_VZ};
    tile_prologue<S, T, G::NT>(sm, bar, maps, field, tl, sh, a.shots, cs, coefs);
    const T *sVx = S::tile(sm, 0), *sVz = S::tile(sm, 1);
    e2d_stress_tile<T, MODE, TX, TZ, RZ, ADJ>(a, sh, tl, sVx, sVz, cs, pt, bar, err);
}

// ---------------------------------------------------------------- sources and receivers
// One CTA per shot.  Injection first (lib/waves.cpp:407-497, 2085-2174), then,
// after a CTA barrier, recording (lib/waves.cpp:500-595, 2178-2288) of the same step.
// A few thousand values at most, so the chain of dependent loads is what it costs: the
// descriptors come to shared memory in one round trip, a thread's first injection point
// and first trace are read, but for the wavefields and samples, before the wait for the
// kernels ahead, and sets that inject into different fields share one pass.  Mean launch of a 16-shot gradient whose adjoint injects 301 traces a shot:
// 9.9 -> 5.8 us on B200; of one shot with one source 4.4 us before and after.

// What recording a trace needs beside the wavefields.
template <typename T>
struct RecPoint {
    const RecSet<T> *q;
    int tr, p;
    T w[4];
    // trace k of all the sets in a row; p = -1: none
    __device__ __forceinline__ void load(const InjRec<T> &pl, int k)
    {
        p = -1;
        for (int set = 0; set < pl.nrecsets; set++) {
            q = &pl.rec[set];
            if (q->kind == REC_NONE) continue;
            if (k < q->nrec) {
                tr = k;
                p = q->pt[tr];
#pragma unroll
                for (int c = 0; c < 4; c++) w[c] = q->w[4 * tr + c];
                return;
            }
            k -= q->nrec;
        }
    }
};

// Injection point: what it needs beside the wavefields and the wavelet (its first
// contribution among it), then the injection, contributions in the reference's order.
template <typename T, int MODE>
struct InjPoint {
    const InjSet<T> *q;
    int p, c0, c1, tr;
    T wx, wz, mod;
    __device__ __forceinline__ void load(const Shot2D<T> &sh, const InjSet<T> &set, int j)
    {
        q = &set;
        p = q->pt[j];
        c0 = q->start[j];
        c1 = q->start[j + 1];
        tr = q->trace[c0];
        wx = q->wx[c0];
        wz = q->wz[c0];
        const int m = q->kind == INJ_A2_P ? M_L : q->kind == INJ_A2_VX || q->kind == INJ_E2_VX ? M_RX : M_RZ;
        mod = q->kind == INJ_E2_P ? T(0) : sh.m[m][p];
    }
    __device__ __forceinline__ void inject(const Shot2D<T> &sh, int nt, int it, T dt) const
    {
        using A = Ar<T, MODE == MODE_FAST ? MODE_FAST : MODE_IEEE>;
        if (q->kind == INJ_E2_P) {
            T sxx = sh.f[E2_SXX][p], szz = sh.f[E2_SZZ][p];
            for (int c = c0; c < c1; c++) {
                const T w = q->wav[(long)(c == c0 ? tr : q->trace[c]) * nt + it];
                const T s = A::mul(A::mul(A::mul(dt, w), c == c0 ? wx : q->wx[c]), c == c0 ? wz : q->wz[c]);
                sxx = A::sub(sxx, s);
                szz = A::sub(szz, s);
            }
            sh.f[E2_SXX][p] = sxx;
            sh.f[E2_SZZ][p] = szz;
            return;
        }
        T *F;
        switch (q->kind) {
        case INJ_A2_P: F = sh.f[A2_P]; break;
        case INJ_A2_VX: F = sh.f[A2_VX]; break;
        case INJ_A2_VZ: F = sh.f[A2_VZ]; break;
        case INJ_E2_VX: F = sh.f[E2_VX]; break;
        default: F = sh.f[E2_VZ]; break;
        }
        T v = F[p];
        const T dm = A::mul(dt, mod);
        for (int c = c0; c < c1; c++) {
            const T w = q->wav[(long)(c == c0 ? tr : q->trace[c]) * nt + it];
            v = A::add(v, A::mul(A::mul(A::mul(dm, w), c == c0 ? wx : q->wx[c]), c == c0 ? wz : q->wz[c]));
        }
        F[p] = v;
    }
};
// Point k of all the sets in a row: its set, and k made its index there.
template <typename T>
__device__ __forceinline__ const InjSet<T> &inj_set_of(const InjRec<T> &pl, int &k)
{
    int set = 0;
    while (pl.inj[set].kind == INJ_NONE || k >= pl.inj[set].ninj) {
        k -= pl.inj[set].kind == INJ_NONE ? 0 : pl.inj[set].ninj;
        set++;
    }
    return pl.inj[set];
}

template <typename T, int MODE>
__global__ void __launch_bounds__(1024) inject_record_2d(const Shot2D<T> *shots, const InjRec<T> *plans, T dt,
                                                         int it_base, const int *it_dev)
{
    using A = Ar<T, MODE == MODE_FAST ? MODE_FAST : MODE_IEEE>;
    __shared__ Shot2D<T> sh;
    __shared__ InjRec<T> pl;
    stage_words(sh, shots + blockIdx.x, threadIdx.x, blockDim.x);
    stage_words(pl, plans + blockIdx.x, threadIdx.x, blockDim.x);
    __syncthreads();
    int nrec = 0, ninj = 0;
    for (int set = 0; set < pl.nrecsets; set++) nrec += pl.rec[set].kind == REC_NONE ? 0 : pl.rec[set].nrec;
    // sets that touch the same field add in set order; others share a pass
    bool apart = true;
    for (int a = 0; a < pl.ninjsets; a++) {
        ninj += pl.inj[a].kind == INJ_NONE ? 0 : pl.inj[a].ninj;
        for (int b = 0; b < a; b++) apart = apart && (pl.inj[a].kind != pl.inj[b].kind || pl.inj[a].kind == INJ_NONE);
    }
    RecPoint<T> r;
    r.p = -1;
    if ((int)threadIdx.x < nrec) r.load(pl, threadIdx.x);
    InjPoint<T, MODE> q;
    if (apart && (int)threadIdx.x < ninj) {
        int j = threadIdx.x;
        const InjSet<T> &set = inj_set_of(pl, j);
        q.load(sh, set, j);
    }
    pdl_wait();
    pdl_trigger();
    const int it_step = it_base + (it_dev ? *it_dev : 0);
    const int it = pl.rev ? pl.nt - 1 - it_step : it_step;
    const int gate = pl.rec_gate ? *pl.rec_gate : 1;
    T acc = r.p >= 0 ? r.q->out[(long)r.tr * pl.nt + it] : T(0);
    if (apart) {
        for (int k = threadIdx.x; k < ninj; k += blockDim.x) {
            if (k != (int)threadIdx.x) {
                int j = k;
                const InjSet<T> &set = inj_set_of(pl, j);
                q.load(sh, set, j);
            }
            q.inject(sh, pl.nt, it, dt);
        }
    } else {
        for (int set = 0; set < pl.ninjsets; set++) {
            if (set > 0) __syncthreads();
            if (pl.inj[set].kind == INJ_NONE) continue;
            for (int j = threadIdx.x; j < pl.inj[set].ninj; j += blockDim.x) {
                q.load(sh, pl.inj[set], j);
                q.inject(sh, pl.nt, it, dt);
            }
        }
    }
    if (nrec == 0 || gate == 0) return;
    __syncthreads();
    const int off[4] = {0, 1, sh.pitch, sh.pitch + 1};
    for (int k = threadIdx.x; k < nrec; k += blockDim.x) {
        if (k != (int)threadIdx.x) {
            r.load(pl, k);
            acc = r.p >= 0 ? r.q->out[(long)r.tr * pl.nt + it] : T(0);
        }
        if (r.p < 0) continue;
        const RecSet<T> &q = *r.q;
        const int p = r.p;
        const T wx[4] = {r.w[0], r.w[1], r.w[0], r.w[1]}, wz[4] = {r.w[2], r.w[2], r.w[3], r.w[3]};
        if (q.kind == REC_E2_P) {
            // (1./2.)*xtri*ytri*F/factor is evaluated in double by the reference and
            // added to the T-typed trace sample (lib/waves.cpp:2238-2239)
            const double fac = (double)q.factor[r.tr];
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const double w = __dmul_rn(__dmul_rn(0.5, (double)wx[c]), (double)wz[c]);
                acc = (T)__dadd_rn((double)acc, __ddiv_rn(__dmul_rn(w, (double)sh.f[E2_SXX][p + off[c]]), fac));
                acc = (T)__dadd_rn((double)acc, __ddiv_rn(__dmul_rn(w, (double)sh.f[E2_SZZ][p + off[c]]), fac));
            }
        } else if (q.kind == REC_E2_PSUM) {
#pragma unroll
            for (int c = 0; c < 4; c++)
                acc = A::add(acc, A::mul(A::mul(wx[c], wz[c]), A::add(sh.f[E2_SXX][p + off[c]], sh.f[E2_SZZ][p + off[c]])));
        } else {
            const T *F;
            switch (q.kind) {
            case REC_A2_P: F = sh.f[A2_P]; break;
            case REC_A2_VX: F = sh.f[A2_VX]; break;
            case REC_A2_VZ: F = sh.f[A2_VZ]; break;
            case REC_E2_VX: F = sh.f[E2_VX]; break;
            default: F = sh.f[E2_VZ]; break;
            }
#pragma unroll
            for (int c = 0; c < 4; c++) acc = A::add(acc, A::mul(A::mul(wx[c], wz[c]), F[p + off[c]]));
        }
        q.out[(long)r.tr * pl.nt + it] = acc;
    }
}

static __global__ void advance_counter(int *it_dev, int by)
{
    if (threadIdx.x == 0 && blockIdx.x == 0) *it_dev += by;
}

static __global__ void set_counter(int *it_dev, int value)
{
    if (threadIdx.x == 0 && blockIdx.x == 0) *it_dev = value;
}

// ---------------------------------------------------------------- launchers
template <typename T, int MODE, int TX, int TZ, int RZ, int MINB>
cudaError_t launch_2d_cfg(int physics, int half, int flags, const Step2DArgs<T> &a, const CoefSet<T> *coefs,
                          const CUtensorMap *maps, int *err, int grid, cudaStream_t st)
{
    using G = Geo2D<T, TX, TZ, RZ>;
    auto launch = [&](auto k, size_t smem, SmemLimit &limit) {
        const cudaError_t e = limit.raise(k, smem);
        return e != cudaSuccess ? e : launch_pdl(k, grid, G::NT, smem, st, a, coefs, maps, err);
    };
    static SmemLimit av, as, ev, es, ev_adj, es_adj;
    if (physics == PHYS_A2D) {
        if (half == 0) return launch(a2d_velocity<T, MODE, TX, TZ, RZ, MINB>, SmemA2V<T, TX, TZ>::bytes(), av);
        return launch(a2d_stress<T, MODE, TX, TZ, RZ, MINB>, SmemA2S<T, TX, TZ>::bytes(), as);
    }
    if (flags & LAUNCH_ADJ) {
        if (half == 0) return launch(e2d_velocity<T, MODE, TX, TZ, RZ, MINB, true>, SmemE2V<T, TX, TZ, true>::bytes(), ev_adj);
        return launch(e2d_stress<T, MODE, TX, TZ, RZ, MINB, true>, SmemE2S<T, TX, TZ>::bytes(), es_adj);
    }
    if (half == 0) return launch(e2d_velocity<T, MODE, TX, TZ, RZ, MINB, false>, SmemE2V<T, TX, TZ, false>::bytes(), ev);
    return launch(e2d_stress<T, MODE, TX, TZ, RZ, MINB, false>, SmemE2S<T, TX, TZ>::bytes(), es);
}

}  // namespace rsgpu
