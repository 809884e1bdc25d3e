// fw_kernels.cu -- sm_103a kernels of the FUNWAVE-TVD SSP-RK3 stage.
//
// Every kernel reproduces one or more of the reference's Fortran units on
// the device-resident state (layout in fw_internal.h).  Index ranges,
// in-place update orders and stale-value semantics follow the reference:
//   - ghost cells hold exactly what EXCHANGE / EXCHANGE_DISPERSION leave
//     (PHI_COLL order: periodic copy, x mirror on interior rows, y mirror on
//     all columns; bc.F:631-1272), including the periodic corner cells that
//     keep the value of the x-ghost cell they copy from before that cell is
//     refilled;
//   - BOUNDARY_CONDITION's overlapping dry-face writes (bc.F:214-293) are
//     resolved per face by the write that comes last in the reference's loop;
//   - UPDATE_MASK is a Jacobi update (masks.F:75-143) with the order-
//     dependent Depthx/Depthy reset (masks.F:152-161) resolved per face;
//   - the breaking AGE sweep (breaker.F:149-229) is an in-place Gauss-Seidel
//     sweep; it is reproduced exactly by evaluating every cell whose result
//     does not depend on its neighbours in parallel, then iterating the rest
//     (cells with AGE = 0 and Cbrk2 <= ETAt < Cbrk1) to the fixed point of
//     the sweep's acyclic dependency graph.
// T is the storage and arithmetic type of the bulk fields (double or
// float); the tridiagonal u/v recovery always runs in double.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <algorithm>
#include <cstring>
#include <initializer_list>
#include <type_traits>

#include "fw_internal.h"
#include "fw_tc.cuh"

namespace fw {

#define IDX(i, j) ((size_t)(i) + (size_t)(j) * (size_t)g.pitch)
// in 32 bits (fw_create keeps a plane below 2^31 cells): fewer instructions and
// registers an address where a kernel reads one cell of many planes
// (2048 x 2048: k_post_mask_break 62 -> 52 us, k_disp_a 60 -> 57); the stencils of k_disp_b and
// k_update are faster with IDX (115 and 128 us, 131 and 132 with this)
#define IDI(i, j) ((i) + (j) * g.pitch)

// pi as the reference stores it: a default-REAL literal (mod_param.F:71)
constexpr double PI_SP = (double)(float)3.141592653;
// the default-REAL literal 4.004 of SigWaveHeight (mixing.F:244)
constexpr double C4004_SP = (double)(float)4.004;
constexpr double GRAV = 9.81;
constexpr double SMALL = 0.000001;
constexpr double LARGE = 999999.0;

// bring the cache line of p into L1 (no value, no register): later loads of
// inputs that the compiler may not move above earlier stores then hit L1
__device__ __forceinline__ void prefetch_l1(const void *p) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}
// a load of an array that the kernel does not write: the read-only data
// path, which also frees the compiler to issue it before the kernel's
// stores (the Fields pointers could otherwise alias them)
template <typename X> __device__ __forceinline__ X ro(const X *p) { return __ldg(p); }
// the same of element id; in the mixed path the offset in bytes has 32 bits too,
// so that the address is a uniform base and one register (a float plane of 4
// GiB would need an arena of more than 288 GiB)
template <typename X> __device__ __forceinline__ X ro(const X *p, int id) {
    if constexpr (sizeof(X) <= 4) return __ldg((const X *)((const char *)p + (unsigned)id * (unsigned)sizeof(X)));
    else return __ldg(p + id);
}

__device__ __forceinline__ double fsqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float fsqrt(float x) { return sqrtf(x); }
__device__ __forceinline__ double fabs_(double x) { return fabs(x); }
__device__ __forceinline__ float fabs_(float x) { return fabsf(x); }
__device__ __forceinline__ double fcopysign(double a, double b) { return copysign(a, b); }
__device__ __forceinline__ float fcopysign(float a, float b) { return copysignf(a, b); }
__device__ __forceinline__ double fexp(double x) { return exp(x); }
__device__ __forceinline__ float fexp(float x) { return expf(x); }
__device__ __forceinline__ double fsin(double x) { return sin(x); }
__device__ __forceinline__ float fsin(float x) { return sinf(x); }
__device__ __forceinline__ double fcos(double x) { return cos(x); }
__device__ __forceinline__ float fcos(float x) { return cosf(x); }
__device__ __forceinline__ double ftanh(double x) { return tanh(x); }
__device__ __forceinline__ float ftanh(float x) { return tanhf(x); }
__device__ __forceinline__ double fatan2(double y, double x) { return atan2(y, x); }
__device__ __forceinline__ float fatan2(float y, float x) { return atan2f(y, x); }

// a constant of the grid block in the kernel's precision: the double member
// in FP64, its float copy f_<name> in the mixed path (no FP64 work there)
#define GC(name) (sizeof(T) == sizeof(double) ? (T)g.name : (T)g.f_##name)
// DT of the current step in the kernel's precision
#define DTV (sizeof(T) == sizeof(double) ? (T)f.dsc[S_DT] : (T)f.fsc[FS_DT])

// a 0/1 mask byte as a real, by a select instead of an integer-to-float
// conversion instruction
template <typename T> __device__ __forceinline__ T m2r(int m) { return m ? (T)1 : (T)0; }
// a small integer (|k| < 2^22) as a real; in float exactly, by placing k in
// the mantissa of 1.5*2^23 and subtracting that constant
template <typename T> __device__ __forceinline__ T i2r(int k) {
    if constexpr (sizeof(T) == sizeof(double)) return (T)k;
    else return __int_as_float(0x4B400000 + k) - 12582912.0f;
}
template <typename T> __device__ __forceinline__ T tmax(T a, T b) { return a > b ? a : b; }
template <typename T> __device__ __forceinline__ T tmin(T a, T b) { return a < b ? a : b; }

// ---------------------------------------------------------------------------
// FP64 arithmetic beside the FP64 pipe.  GB300 issues double operations at
// 1/64 of the float rate and integer ones beside them, so comparisons,
// absolute values and doublings of doubles are done on their bits, and
// quotients by a divisor whose reciprocal is at hand take one product and two
// fused operations.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long dbits(double x) { return (unsigned long long)__double_as_longlong(x); }
__device__ __forceinline__ double dfrom(unsigned long long b) { return __longlong_as_double((long long)b); }
constexpr unsigned long long D_SIGN = 1ull << 63, D_INF = 0x7ffull << 52;
__device__ __forceinline__ unsigned long long dmag(double x) { return dbits(x) & ~D_SIGN; }

// a / b rounded to nearest, with y = RN(1/b): q = RN(a y), r = a - b q
// (exact), RN(q + r y) (Markstein, IBM J. Res. Dev. 34 (1990): correctly
// rounded when y is, and nothing under- or overflows).  |b| lies in
// [2^-300, 2^300] (the callers' spacings, steps and coefficients); an a
// outside [2^-500, 2^500], zero apart, takes the division.
__device__ __forceinline__ double div_rcp(double a, double b, double y) {
    const unsigned long long m = dmag(a);
    if (m - ((1023ull - 500) << 52) >= (1000ull << 52)) {
        if (m == 0) return dfrom(dbits(a) ^ (dbits(b) & D_SIGN));
        return a / b;
    }
    const double q = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(-q, b, a), y, q);
}

// whether a b lies in div_rcp's range
__device__ __forceinline__ bool div_rcp_ok(double b) {
    const unsigned long long m = dmag(b);
    return m >= ((1023ull - 300) << 52) && m <= ((1023ull + 300) << 52);
}
// a / b for any b; y = RN(1/b)
__device__ __forceinline__ double div_any(double a, double b, double y) {
    const bool ok = div_rcp_ok(b);  // of b alone: once for all quotients by it
    const unsigned long long m = dmag(a);
    if (m - ((1023ull - 500) << 52) >= (ok ? 1000ull << 52 : 0)) {
        if (m == 0 && ok) return dfrom(dbits(a) ^ (dbits(b) & D_SIGN));
        return a / b;
    }
    const double q = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(-q, b, a), y, q);
}
// x / b for a constant b of the run whose reciprocal y is at hand: FP64 by
// div_any, which rounds as the division; the mixed path multiplies
__device__ __forceinline__ double over(double x, double b, double y) { return div_any(x, b, y); }
__device__ __forceinline__ float over(float x, float, float y) { return x * y; }
// the larger of x and a positive b (b for a NaN, as tmax), on the bits in
// FP64: doubles order like their bits against a positive one
__device__ __forceinline__ double max_pos(double x, double b) {
    const long long m = __double_as_longlong(x);
    return m > __double_as_longlong(b) && m <= (long long)D_INF ? x : b;
}
__device__ __forceinline__ float max_pos(float x, float b) { return x > b ? x : b; }
// a - 2 b: the product is exact, so FP64's fused operation rounds as the two
__device__ __forceinline__ double sub2(double a, double b) { return __fma_rn(-2.0, b, a); }
__device__ __forceinline__ float sub2(float a, float b) { return a - 2.0f * b; }

// ---------------------------------------------------------------------------
// exchange source of a ghost cell (PHI_COLL, serial branches)
// ---------------------------------------------------------------------------
__device__ __forceinline__ int mirror_x(const Grid &g, int i) {
    return i < g.ib ? 2 * g.ib - 1 - i : (i > g.ie ? 2 * g.ie + 1 - i : i);
}
__device__ __forceinline__ int mirror_y(const Grid &g, int j) {
    return j < g.jb ? 2 * g.jb - 1 - j : (j > g.je ? 2 * g.je + 1 - j : j);
}
// periodic-y source row of a ghost row (bc.F:735-740)
__device__ __forceinline__ int period_y(const Grid &g, int j) {
    return j < g.jb ? j + g.je - 2 : (j > g.je ? j - g.je + 2 : j);
}

// ---------------------------------------------------------------------------
// Lines ahead: a kernel whose threads each read one cell of many planes has
// too few of those reads in flight (its registers bound the blocks on an SM)
// to cover the memory's latency.  Its threads therefore also bring to the L2,
// one line each, the lines that the block `dist` places later reads; that
// block's loads then wait for the L2 only.
// Mixed 2048 x 2048: k_update 146 -> 128 us, k_disp_a 74 -> 60,
// k_post_mask_break 68 -> 62, k_exchange 35 -> 33 and at a step's begin 94 ->
// 86.  The distance matters little between one and four blocks per SM (with
// twice the resident blocks the gain is gone); k_disp_b and the fluxes, bound
// by their issue, gain nothing.
// ---------------------------------------------------------------------------
struct Ahead {
    const void *p[28];
    int n;       // planes (0: none)
    int dx, dy;  // the later block: columns and rows of blocks from this one
    int lx, ll;  // log2 of a block's lines of a plane: in a row, in all
};
// dist: blocks ahead in a grid of nbx columns of blocks b; from min_cells cells
// on, and for blocks of a power of two of lines (the thread's line then needs
// no division)
template <typename T>
static Ahead ahead_of(const Grid &g, dim3 b, int nbx, long long min_cells, int dist, std::initializer_list<const T *> planes) {
    Ahead a{};
    const unsigned nx = (b.x + 31) / 32, lines = nx * b.y;
    if (sizeof(T) != sizeof(float) || (long long)g.Mloc * g.Nloc < min_cells || (nx & (nx - 1)) || (lines & (lines - 1)))
        return a;
    for (const T *q : planes) a.p[a.n++] = q;
    a.dx = dist % nbx;
    a.dy = dist / nbx;
    while (1u << a.lx < nx) a.lx++;
    while (1u << a.ll < lines) a.ll++;
    return a;
}
// blocks of blockDim.x x blockDim.y cells from column 0 and row j0 on; by: the
// block's row
template <typename T>
__device__ __forceinline__ void prefetch_ahead(const Grid &g, const Ahead &a, int by, int j0) {
    if constexpr (sizeof(T) == sizeof(float)) {
        if (a.n == 0) return;
        int bx = blockIdx.x + a.dx;
        by += a.dy;
        if (bx >= (int)gridDim.x) {
            bx -= gridDim.x;
            by++;
        }
        const int i0 = bx * blockDim.x;
        j0 += by * blockDim.y;
        for (int t = threadIdx.x + threadIdx.y * blockDim.x; t < a.n << a.ll; t += blockDim.x * blockDim.y) {
            const int q = t >> a.ll, r = t & ((1 << a.ll) - 1), i = i0 + (r & ((1 << a.lx) - 1)) * 32, j = j0 + (r >> a.lx);
            if (i < g.Mloc && j < g.Nloc)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const T *>(a.p[q]) + IDI(i, j)));
        }
    }
}

// ---------------------------------------------------------------------------
// CAL_DISPERSION, part 1 (dispersion.F:62-289): masked derivatives at the
// exchange source of every cell, combined into the four sums the rest of
// the unit uses, plus ETAx/ETAy (exchanged) and ETAT.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) k_disp_a(Grid g, Fields<T> f, Ahead ah) {
    prefetch_ahead<T>(g, ah, blockIdx.y, 0);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= g.Mloc || j >= g.Nloc) return;
    const T DX = GC(DX), DY = GC(DY), mdf = GC(min_depth_frc);
    const int id = IDI(i, j);
    // ETAT from the previous stage's face fluxes (dispersion.F:103-119)
    if (i <= g.Mloc - 2 && j <= g.Nloc - 2) {
        if constexpr (sizeof(T) == sizeof(double))
            f.ETAT[id] = over(-(ro(f.P + (IDI(i + 1, j))) - ro(f.P + (id))), DX, (T)g.rdx) -
                         over(ro(f.Q + (IDI(i, j + 1))) - ro(f.Q + (id)), DY, (T)g.rdy);
        else
            f.ETAT[id] = -(ro(f.P + (IDI(i + 1, j))) - ro(f.P + (id))) * GC(rdx) - (ro(f.Q + (IDI(i, j + 1))) - ro(f.Q + (id))) * GC(rdy);
    }

    const bool gx = (i < g.ib) || (i > g.ie);
    const bool gy = (j < g.jb) || (j > g.je);
    const int si = mirror_x(g, i);
    int sj = j;
    T sy3 = (T)1;  // sign of VTYPE 3 fields in a y ghost
    bool stale = false;
    if (gy) {
        if (g.periodic) {
            sj = period_y(g, j);
            stale = gx;  // periodic corner: keeps the pre-exchange value
        } else {
            sj = mirror_y(g, j);
            sy3 = (T)-1;
        }
    }
    const T sx2 = gx ? (T)-1 : (T)1;  // sign of VTYPE 2 fields in an x ghost

    const T m9 = m2r<T>(ro(f.MASK9 + (IDI(si, sj))));
    const bool wall = (si == g.ib) || (si == g.ie) || (sj == g.jb) || (sj == g.je);
#define LU(a, b) ro(f.U + (IDI(si + (a), sj + (b))))
#define LV(a, b) ro(f.V + (IDI(si + (a), sj + (b))))
#define LDU(a, b) (max_pos(ro(f.Depth + (IDI(si + (a), sj + (b)))), mdf) * LU(a, b))
#define LDV(a, b) (max_pos(ro(f.Depth + (IDI(si + (a), sj + (b)))), mdf) * LV(a, b))
    // FP64: the reference's divisions; mixed: reciprocal constants
    constexpr bool EXACT = sizeof(T) == sizeof(double);
    const T rdx2 = (T)g.f_rdx2, rdy2 = (T)g.f_rdy2, rdxy4 = (T)g.f_rdxy4;
#define QX(x) div_any((double)(x), g.DX, g.rdx)
#define QY(x) div_any((double)(x), g.DY, g.rdy)
#define DXX(F) (EXACT ? (T)(QX(QX(sub2(F(1, 0), F(0, 0)) + F(-1, 0))) * m9) \
                      : ((F(1, 0) - (T)2 * F(0, 0) + F(-1, 0)) * rdx2 * m9))
#define DYY(F) (EXACT ? (T)(QY(QY(sub2(F(0, 1), F(0, 0)) + F(0, -1))) * m9) \
                      : ((F(0, 1) - (T)2 * F(0, 0) + F(0, -1)) * rdy2 * m9))
#define DXY(F)                                                                                      \
    (wall ? (T)0                                                                                    \
          : (EXACT ? (T)(QX((QY((F(1, 1) - F(1, -1)) / (T)2) - QY((F(-1, 1) - F(-1, -1)) / (T)2)) / (T)2) * m9) \
                   : (((F(1, 1) - F(1, -1)) - (F(-1, 1) - F(-1, -1))) * rdxy4 * m9)))
    const T Uxx = DXX(LU), Vyy = DYY(LV), Uxy = DXY(LU), Vxy = DXY(LV);
    const T DUxx = DXX(LDU), DVyy = DYY(LDV), DUxy = DXY(LDU), DVxy = DXY(LDV);
#undef LU
#undef LV
#undef LDU
#undef LDV
#undef DXX
#undef DYY
#undef DXY
    if constexpr (sizeof(T) == sizeof(double)) {
        // FP64: keep every exchanged term (VTYPE 2: Uxx DUxx; 3: Vyy DVyy;
        // 1: the cross derivatives), as EXCHANGE_DISPERSION leaves them
        f.Uxx[id] = sx2 * Uxx;
        f.DUxx[id] = sx2 * DUxx;
        f.Vyy[id] = sy3 * Vyy;
        f.DVyy[id] = sy3 * DVyy;
        f.Uxy[id] = Uxy;
        f.Vxy[id] = Vxy;
        f.DUxy[id] = DUxy;
        f.DVxy[id] = DVxy;
    } else {
        f.A[id] = sx2 * Uxx + Vxy;
        f.B[id] = sx2 * DUxx + DVxy;
        f.C[id] = Uxy + sy3 * Vyy;
        f.E[id] = DUxy + sy3 * DVyy;
    }
    // ETAx, ETAy: computed on the interior and exchanged only when Gamma2 > 0
    // (bc.F:395-398); without Gamma2 the ghosts keep their old values
    const bool exch = g.has_g2 != 0;
    if (exch || (g.show_breaking && !gx && !gy)) {
        const T dex = ro(f.Eta + (IDI(si + 1, sj))) - ro(f.Eta + (IDI(si - 1, sj)));
        const T dey = ro(f.Eta + (IDI(si, sj + 1))) - ro(f.Eta + (IDI(si, sj - 1)));
        const T ex = EXACT ? (T)(QX(dex) / 2.0 * m9) : dex * (T)g.f_hdx * m9;
        const T ey = EXACT ? (T)(QY(dey) / 2.0 * m9) : dey * (T)g.f_hdy * m9;
        if (!stale) {
            if (exch && g.periodic && gx && !gy) {
                // the periodic copy (bc.F:735-740) runs before the x mirror:
                // a corner cell receives this x-ghost cell's previous value
                if (j >= g.je - 2) {
                    f.ETAx[IDI(i, j - (g.je - 2))] = f.ETAx[id];
                    f.ETAy[IDI(i, j - (g.je - 2))] = f.ETAy[id];
                }
                if (j <= g.jb + 2) {
                    f.ETAx[IDI(i, j + g.je - 2)] = f.ETAx[id];
                    f.ETAy[IDI(i, j + g.je - 2)] = f.ETAy[id];
                }
            }
            f.ETAx[id] = sx2 * ex;
            f.ETAy[id] = sy3 * ey;
        }
    }
}

// ---------------------------------------------------------------------------
// CAL_DISPERSION, part 2 (dispersion.F:293-503): U4, V4 on every cell;
// U1p, V1p and U1pp+U2+U3, V1pp+V2+V3 on the interior.
// ---------------------------------------------------------------------------
// In FP64 the pipe is the bound (81 % busy): constant divisors divide through
// their reciprocals, the time derivatives are taken once per cell of a tile
// and the constants come evaluated (701 x 937: 1412 -> 726 us; k_disp_a the
// same way 438 -> 252, k_update 555 -> 372).
// the combinations of Beta_1 and Beta_2 that k_disp_b multiplies by, evaluated
// in double in the reference's order (the FP64 mode's; the host's operations
// round as the device's)
struct DispK {
    double c1, c2, c3, c4, c5, c6, c7, c8, c9, c10, c11, c12, c13;
};
static DispK disp_k(const Grid &g) {
    const double B1 = g.Beta_1, B2 = g.Beta_2;
    // one operation to a statement: nothing to contract
    auto mul = [](double a, double b) { volatile double r = a * b; return (double)r; };
    DispK k;
    k.c8 = mul(B1, B1);
    k.c13 = mul(mul(0.5, B1), B1);
    volatile double t = 1.0 / 3.0 - B1;
    k.c1 = t + k.c13;
    k.c2 = B1 - 0.5;
    t = 1.0 / 6.0 - B1;
    k.c3 = t + k.c8;
    k.c4 = mul(mul(0.5, B1), B1) - 1.0 / 6.0;
    const double m = 1.0 - B1;
    k.c5 = mul(mul(0.5, m), m);
    k.c6 = B1 - 1.0;
    k.c7 = mul(B1, m);
    k.c9 = mul(m, m);
    k.c10 = k.c8 - 1.0;
    k.c11 = mul(0.5, k.c10);
    k.c12 = mul(B2, B2);
    return k;
}
// shared memory of k_disp_b: the FP64 tile's four planes
template <typename T> static size_t disp_b_smem(dim3 b) {
    return sizeof(T) == sizeof(double) ? (size_t)4 * (b.x + 2) * (b.y + 2) * sizeof(double) : 0;
}

template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == sizeof(float) ? 4 : 1) k_disp_b(Grid g, Fields<T> f, DispK dk) {
    constexpr bool EXACT = sizeof(T) == sizeof(double);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const T mdf = GC(min_depth_frc), DT = DTV;
    extern __shared__ double dsm[];
    // FP64: the time derivatives of the tile's cells and of the ring around
    // it, and their products with the depth, once per cell
    const int tw = blockDim.x + 2, tc = tw * (blockDim.y + 2);
    const int tq = (threadIdx.x + 1) + (threadIdx.y + 1) * tw;
    if constexpr (EXACT) {
        if (g.has_g2) {
            const double rdt = __drcp_rn((double)DT);
            for (int q = threadIdx.x + threadIdx.y * blockDim.x; q < tc; q += blockDim.x * blockDim.y) {
                const int a = (int)(blockIdx.x * blockDim.x) - 1 + q % tw, c = (int)(blockIdx.y * blockDim.y) - 1 + q / tw;
                if (a < 0 || a >= g.Mloc || c < 0 || c >= g.Nloc) continue;
                const size_t id = IDX(a, c);
                const double dep = max_pos((double)f.Depth[id], (double)mdf);
                const double ut = div_any((double)(f.U[id] - f.U0[id]), (double)DT, rdt);
                const double vt = div_any((double)(f.V[id] - f.V0[id]), (double)DT, rdt);
                dsm[q] = ut;
                dsm[tc + q] = vt;
                dsm[2 * tc + q] = dep * ut;
                dsm[3 * tc + q] = dep * vt;
            }
            __syncthreads();
        }
    }
    if (i >= g.Mloc || j >= g.Nloc) return;
    const size_t id = IDX(i, j);
    const T DX = GC(DX), DY = GC(DY);
    const T B1 = GC(Beta_1), B2 = GC(Beta_2), g2 = GC(gamma2), b2 = GC(b2);
    const T one = (T)1, two = (T)2, half = (T)0.5;
    const T D = f.Depth[id], reta = f.Eta[id], m9 = m2r<T>(f.MASK9[id]);
    // the combinations of Beta_1 and Beta_2: FP64 reads them (each would cost
    // every thread FP64 operations), the mixed path computes them
#define DK(name, expr) (EXACT ? (T)dk.name : (T)(expr))
    const T c1 = DK(c1, one / (T)3 - B1 + half * B1 * B1), c2 = DK(c2, B1 - one / two);
    const T c3 = DK(c3, one / (T)6 - B1 + B1 * B1), c4 = DK(c4, one / two * B1 * B1 - one / (T)6);
    const T c5 = DK(c5, half * (one - B1) * (one - B1)), c6 = DK(c6, B1 - one), c7 = DK(c7, B1 * (one - B1));
    const T c8 = DK(c8, B1 * B1), c9 = DK(c9, (one - B1) * (one - B1)), c10 = DK(c10, B1 * B1 - one);
    const T c11 = DK(c11, half * (B1 * B1 - one)), c12 = DK(c12, B2 * B2), c13 = DK(c13, half * B1 * B1);
#undef DK
    T a, b, c, e;
    if constexpr (EXACT) {
        a = f.Uxx[id] + f.Vxy[id];
        b = f.DUxx[id] + f.DVxy[id];
        c = f.Uxy[id] + f.Vyy[id];
        e = f.DUxy[id] + f.DVyy[id];
    } else {
        a = f.A[id];
        b = f.B[id];
        c = f.C[id];
        e = f.E[id];
    }
    T u4 = c1 * D * D * a + c2 * D * b;
    T v4 = c1 * D * D * c + c2 * D * e;
    if (g.has_g2) {
        const T ken1 = c3 * D * reta * B2 +
                       c4 * reta * reta * B2 * B2;
        const T ken2 = c2 * reta * B2;
        u4 = u4 + g2 * m9 * (ken1 * a + ken2 * b);
        v4 = v4 + g2 * m9 * (ken1 * c + ken2 * e);
    }
    f.U4[id] = u4;
    f.V4[id] = v4;
    if (i < g.ib || i > g.ie || j < g.jb || j > g.je) return;

    f.U1p[id] = c5 * D * D * a + c6 * D * b;
    f.V1p[id] = c5 * D * D * c + c6 * D * e;
    if (!g.has_g2) return;

    const T rDT = (T)f.fsc[FS_RDT];
    const T hdx = (T)g.f_hdx, hdy = (T)g.f_hdy;
    const T rdx2 = (T)g.f_rdx2, rdy2 = (T)g.f_rdy2, rdxy4 = (T)g.f_rdxy4;
    const bool wall = (i == g.ib) || (i == g.ie) || (j == g.jb) || (j == g.je);
#define AT(F, a_, b_) f.F[IDX(i + (a_), j + (b_))]
    const T UxxVxy = a, UxyVyy = c, HUxxHVxy = b, HUxyHVyy = e;
    T UxxVxy_x, UxxVxy_y, UxyVyy_x, UxyVyy_y, HUxxHVxy_x, HUxxHVxy_y, HUxyHVyy_x, HUxyHVyy_y;
    if constexpr (EXACT) {
        // (F1(I+1)+F2(I+1)-F1(I-1)-F2(I-1))/2/DX, evaluated left to right
#define DIFF(F1, F2, a1, b1, a2, b2, H) \
    H((AT(F1, a1, b1) + AT(F2, a1, b1) - AT(F1, a2, b2) - AT(F2, a2, b2)) / two)
        UxxVxy_x = DIFF(Uxx, Vxy, 1, 0, -1, 0, QX);
        UxxVxy_y = DIFF(Uxx, Vxy, 0, 1, 0, -1, QY);
        UxyVyy_x = DIFF(Uxy, Vyy, 1, 0, -1, 0, QX);
        UxyVyy_y = DIFF(Uxy, Vyy, 0, 1, 0, -1, QY);
        HUxxHVxy_x = DIFF(DUxx, DVxy, 1, 0, -1, 0, QX);
        HUxxHVxy_y = DIFF(DUxx, DVxy, 0, 1, 0, -1, QY);
        HUxyHVyy_x = DIFF(DUxy, DVyy, 1, 0, -1, 0, QX);
        HUxyHVyy_y = DIFF(DUxy, DVyy, 0, 1, 0, -1, QY);
#undef DIFF
    } else {
        const T hx = (T)g.f_hdx, hy = (T)g.f_hdy;
        UxxVxy_x = (AT(A, 1, 0) - AT(A, -1, 0)) * hx;
        UxxVxy_y = (AT(A, 0, 1) - AT(A, 0, -1)) * hy;
        UxyVyy_x = (AT(C, 1, 0) - AT(C, -1, 0)) * hx;
        UxyVyy_y = (AT(C, 0, 1) - AT(C, 0, -1)) * hy;
        HUxxHVxy_x = (AT(B, 1, 0) - AT(B, -1, 0)) * hx;
        HUxxHVxy_y = (AT(B, 0, 1) - AT(B, 0, -1)) * hy;
        HUxyHVyy_x = (AT(E, 1, 0) - AT(E, -1, 0)) * hx;
        HUxyHVyy_y = (AT(E, 0, 1) - AT(E, 0, -1)) * hy;
    }
    const T rh = D;
    const T rhx = EXACT ? (T)QX((AT(Depth, 1, 0) - AT(Depth, -1, 0)) / two) : (AT(Depth, 1, 0) - AT(Depth, -1, 0)) * hdx;
    const T rhy = EXACT ? (T)QY((AT(Depth, 0, 1) - AT(Depth, 0, -1)) / two) : (AT(Depth, 0, 1) - AT(Depth, 0, -1)) * hdy;
    const T ETAx = f.ETAx[id], ETAy = f.ETAy[id], ETAT = f.ETAT[id];
    // first derivatives of U, V, DU, DV (derivatives.F:123-162)
#define FD1X(F) (EXACT ? (T)((QX(F(1, 0) - F(-1, 0)) / 2.0) * m9) : ((F(1, 0) - F(-1, 0)) * hdx) * m9)
#define FD1Y(F) (EXACT ? (T)((QY(F(0, 1) - F(0, -1)) / 2.0) * m9) : ((F(0, 1) - F(0, -1)) * hdy) * m9)
#define LU_(a_, b_) AT(U, a_, b_)
#define LV_(a_, b_) AT(V, a_, b_)
    const T Ux = FD1X(LU_);
    const T Vx = FD1X(LV_);
    const T Uy = FD1Y(LU_);
    const T Vy = FD1Y(LV_);
#undef LU_
#undef LV_
#define DUP(a_, b_) (max_pos(AT(Depth, a_, b_), mdf) * AT(U, a_, b_))
#define DVP(a_, b_) (max_pos(AT(Depth, a_, b_), mdf) * AT(V, a_, b_))
    const T DUx = FD1X(DUP);
    const T DVy = FD1Y(DVP);
    // time derivatives Ut=(U-U0)/DT (dispersion.F:133-141) and their
    // derivatives; the cross derivatives are zero on the wall rows
#define TSM(k, a_, b_) (T)dsm[(k) * tc + tq + (a_) + (b_) * tw]
#define UT(a_, b_) (EXACT ? TSM(0, a_, b_) : ((AT(U, a_, b_) - AT(U0, a_, b_)) * rDT))
#define VT(a_, b_) (EXACT ? TSM(1, a_, b_) : ((AT(V, a_, b_) - AT(V0, a_, b_)) * rDT))
#define DUT(a_, b_) (EXACT ? TSM(2, a_, b_) : (tmax(AT(Depth, a_, b_), mdf) * UT(a_, b_)))
#define DVT(a_, b_) (EXACT ? TSM(3, a_, b_) : (tmax(AT(Depth, a_, b_), mdf) * VT(a_, b_)))
#define D1X(F) FD1X(F)
#define D1Y(F) FD1Y(F)
#define D2X(F) (EXACT ? (T)(QX(QX(sub2(F(1, 0), F(0, 0)) + F(-1, 0))) * m9) \
                      : ((F(1, 0) - two * F(0, 0) + F(-1, 0)) * rdx2 * m9))
#define D2Y(F) (EXACT ? (T)(QY(QY(sub2(F(0, 1), F(0, 0)) + F(0, -1))) * m9) \
                      : ((F(0, 1) - two * F(0, 0) + F(0, -1)) * rdy2 * m9))
#define D2XY(F)                                                                                          \
    (wall ? (T)0                                                                                         \
          : (EXACT ? (T)(QX((QY((F(1, 1) - F(1, -1)) / two) - QY((F(-1, 1) - F(-1, -1)) / two)) / two) * m9) \
                   : (((F(1, 1) - F(1, -1)) - (F(-1, 1) - F(-1, -1))) * rdxy4 * m9)))
    const T Utx = D1X(UT), Vty = D1Y(VT);
    const T Utxx = D2X(UT), Vtyy = D2Y(VT);
    const T Utxy = D2XY(UT), Vtxy = D2XY(VT);
    const T DUtx = D1X(DUT), DVty = D1Y(DVT);
    const T DUtxx = D2X(DUT), DVtyy = D2Y(DVT);
    const T DUtxy = D2XY(DUT), DVtxy = D2XY(DVT);
#undef D1X
#undef D1Y
#undef D2X
#undef D2Y
#undef D2XY
#undef UT
#undef VT
#undef DUT
#undef DVT
#undef TSM
#undef DUP
#undef DVP
#undef FD1X
#undef FD1Y
    const T Uc = f.U[id], Vc = f.V[id];
#undef AT
    T U1pp = -reta * B2 * ETAx * B2 * (Utx + Vty) - half * reta * reta * B2 * B2 * (Utxx + Vtxy) -
             ETAx * B2 * (DUtx + DVty) - reta * B2 * (DUtxx + DVtxy);
    T V1pp = -reta * B2 * ETAy * B2 * (Utx + Vty) - half * reta * reta * B2 * B2 * (Utxy + Vtyy) -
             ETAy * B2 * (DUtx + DVty) - reta * B2 * (DUtxy + DVtyy);
    T ken1 = c7 * rh * ETAT * B2 - c8 * reta * B2 * ETAT * B2;
    T ken2 = c7 * rh * reta * B2 - c13 * reta * reta * B2 * B2;
    T ken3 = B1 * ETAT * B2;
    T ken4 = B1 * reta * B2;
    U1pp = U1pp - ken1 * UxxVxy - ken2 * (Utxx + Vtxy) + ken3 * HUxxHVxy + ken4 * (DUtxx + DVtxy);
    V1pp = V1pp - ken1 * UxyVyy - ken2 * (Utxy + Vtyy) + ken3 * HUxyHVyy + ken4 * (DUtxy + DVtyy);

    ken1 = c6 * (rhx + ETAx) * B2;
    ken2 = c6 * (rh + reta) * B2;
    ken3 = (c9 * rh * rhx * B2 * B2 - c7 * (rhx * reta * B2 + rh * ETAx * B2) +
            c10 * reta * ETAx * B2 * B2);
    ken4 = (c5 * rh * rh * B2 * B2 - c7 * rh * reta * B2 +
            c11 * reta * reta * B2 * B2);
    const T ken5 = (c9 * rh * rhy * B2 * B2 -
                    c7 * (rhy * reta * B2 + rh * ETAy * B2) + c10 * reta * ETAy * B2 * B2);
    const T U2 = ken1 * (Uc * HUxxHVxy + Vc * HUxyHVyy) +
                 ken2 * (Ux * HUxxHVxy + Uc * HUxxHVxy_x + Vx * HUxyHVyy + Vc * HUxyHVyy_x) +
                 ken3 * (Uc * UxxVxy + Vc * UxyVyy) + ken4 * (Ux * UxxVxy + Uc * UxxVxy_x + Vx * UxyVyy + Vc * UxyVyy_x) +
                 c12 * (DUx + DVy + reta * B2 * (Ux + Vy)) * (HUxxHVxy + ETAx * B2 * (Ux + Vy) + reta * B2 * UxxVxy);
    ken1 = c6 * (rhy + ETAy) * B2;
    const T V2 = ken1 * (Uc * HUxxHVxy + Vc * HUxyHVyy) +
                 ken2 * (Uy * HUxxHVxy + Uc * HUxxHVxy_y + Vy * HUxyHVyy + Vc * HUxyHVyy_y) +
                 ken5 * (Uc * UxxVxy + Vc * UxyVyy) + ken4 * (Uy * UxxVxy + Uc * UxxVxy_y + Vy * UxyVyy + Vc * UxyVyy_y) +
                 c12 * (DUx + DVy + reta * B2 * (Ux + Vy)) * (HUxyHVyy + ETAy * B2 * (Ux + Vy) + reta * B2 * UxyVyy);
    const T omega_0 = Vx - Uy;
    const T omega_1 = (b2 * rhx + B1 * ETAx) * B2 * (HUxyHVyy + (b2 * rh + B1 * reta) * B2 * UxyVyy) -
                      (b2 * rhy + B1 * ETAy) * B2 * (HUxxHVxy + (b2 * rh + B1 * reta) * B2 * UxxVxy);
    ken1 = (c2 * (reta + rh) * B2);
    ken2 = c1 * rh * rh * B2 * B2 + c3 * rh * reta * B2 +
           c4 * reta * reta * B2 * B2;
    const T U3 = -Vc * omega_1 - omega_0 * (ken1 * HUxyHVyy + ken2 * UxyVyy);
    const T V3 = Uc * omega_1 + omega_0 * (ken1 * HUxxHVxy + ken2 * UxxVxy);
    f.Udisp[id] = U1pp + U2 + U3;
    f.Vdisp[id] = V1pp + V2 + V3;
}

#undef QX
#undef QY

// ---------------------------------------------------------------------------
// FLUXES (fluxes.F:52-117): 4th-order MUSCL-TVD (CONSTRUCT_HO_X/Y
// :1531-1754), Zhou wave speeds (:352-439), HLL (:171-194) and
// BOUNDARY_CONDITION (bc.F:53-295), fused per face.
// ---------------------------------------------------------------------------
template <typename T> __device__ __forceinline__ T lim3(T a, T b, T c) {
    if constexpr (sizeof(T) == sizeof(float)) {
        // s * max(0, min(|a|, 2 s b, 2 s c)), s = sign(a): the same value
        // without a branch, except that a zero result may carry the other
        // sign, which the float face values (harmonic means of products
        // tested > 0) never see
        const float s = a >= 0.0f ? 1.0f : -1.0f;
        return s * fmaxf(0.0f, fminf(fminf(fabsf(a), 2.0f * s * b), 2.0f * s * c));
    } else {
        // both arms, then a select: each thread gets the value of its arm
        // (signed zeros included) without the warp splitting on the sign
        const T pos = tmax((T)0, tmin(tmin(a, (T)2 * b), (T)2 * c));
        const T neg = tmin((T)0, tmax(tmax(a, (T)2 * b), (T)2 * c));
        return a >= (T)0 ? pos : neg;
    }
}
// Din(p) from v[0..3] = Vin(p-2..p+1), m[0..3] = MASK(p-2..p+1)
// (fluxes.F:1548-1598).  When any of the four cells is dry the reference
// either limits three equal slopes, which returns TXP2 for each of them, or
// zeroes the limited slopes; both give TXP2 - 1/6*(+0) = TXP2 exactly, so
// the limiter is only evaluated for four wet cells.
template <typename T> __device__ __forceinline__ T ho_din(const T *v, const int *m) {
    const T TXP1 = v[1] - v[0], TXP2 = v[2] - v[1], TXP3 = v[3] - v[2];
    if (!(m[0] && m[1] && m[2] && m[3])) return TXP2;
    const T DVP1 = lim3(TXP1, TXP2, TXP3), DVP2 = lim3(TXP2, TXP3, TXP1), DVP3 = lim3(TXP3, TXP1, TXP2);
    return TXP2 - (T)1 / (T)6 * (DVP3 - (T)2 * DVP2 + DVP1);
}
template <typename T> __device__ __forceinline__ T vl_guard(T t) {
    if (fabs_(t) <= (T)SMALL) t = (T)SMALL * fcopysign((T)1, t);
    return t;
}
template <typename T> __device__ __forceinline__ T vl_phi(T rat) {
    T van = (T)0;
    if (fabs_((T)1 + rat) > (T)SMALL) van = (rat + fabs_(rat)) / ((T)1 + rat);
    return van;
}
template <typename T> __device__ __forceinline__ T hll(T SL, T SR, T FL, T FR, T UL, T UR) {
    if (SL >= (T)0) return FL;
    if (SR <= (T)0) return FR;
    T f = SR * FL - SL * FR + SL * SR * (UR - UL);
    if (fabs_(SR - SL) < (T)SMALL) return f / (T)SMALL;
    return f / (SR - SL);
}
template <typename T> __device__ __forceinline__ T press(T Xi, T Deps, T g3) {
    return (T)0.5 * (T)GRAV * (Xi * Xi * g3 + (T)2 * Xi * Deps);
}

// Limited face values of one field from Din(p-1), Din(p), Din(p+1) and the
// cells p-1, p.  FP64 evaluates the reference's van Leer expressions
// (fluxes.F:1602-1630), including its guard that replaces a slope
// |t| <= SMALL by SMALL*sign(t).  The mixed path uses the equal closed form
// VAN1*TMP1 = VAN2*TMP2 = 2*TMP1*TMP2/(TMP1+TMP2) for TMP1*TMP2 > 0, else 0,
// without the guard (which only adds SMALL-sized corrections, e.g. on still
// water; the closed form needs no guard since TMP1*TMP2 > 0 keeps
// TMP1+TMP2 away from 0).
template <typename T>
__device__ __forceinline__ void ho_lr(T vm1, T v0, T d0, T d1, T d2, T &L, T &R) {
    if constexpr (sizeof(T) == sizeof(double)) {
        T t1 = vl_guard(d0), t2 = vl_guard(d1);
        T van1 = vl_phi(t2 / t1), van2 = vl_phi(t1 / t2);
        L = vm1 + ((T)1 / (T)6) * (van1 * t1 + (T)2 * van2 * t2);
        t1 = vl_guard(d1);
        t2 = vl_guard(d2);
        van1 = vl_phi(t2 / t1);
        van2 = vl_phi(t1 / t2);
        R = v0 - ((T)1 / (T)6) * ((T)2 * van1 * t1 + van2 * t2);
    } else {
        const T t1 = d0, t2 = d1, t3 = d2;
        const T hl = (t1 * t2 > (T)0) ? (T)2 * t1 * t2 / (t1 + t2) : (T)0;
        const T hr = (t2 * t3 > (T)0) ? (T)2 * t2 * t3 / (t2 + t3) : (T)0;
        L = vm1 + (T)0.5 * hl;
        R = v0 - (T)0.5 * hr;
    }
}

// Faces of direction DIR (0: x-faces, 1: y-faces).  A tile is 32 x FY
// faces, FY/8 per thread (by default 32 x 8 x-faces and 32 x 32 y-faces,
// so that the three-cell halo along y is shared by 32 faces; 32 x 16 in
// FP64; fw_autotune may pick another compiled height).  Din of the seven reconstructed fields is
// computed once per cell position into shared memory; each thread then
// finishes its faces: face values, Zhou wave speeds, HLL and the
// boundary/dry-face rules.  Normal velocity is U for x and V for y.
template <typename T, int DIR> constexpr int flux_fy_default() {
    return DIR == 0 ? 8 : (sizeof(T) == sizeof(double) ? 16 : 32);
}

template <typename T, int DIR, int FY_ = flux_fy_default<T, DIR>()> struct FluxTile {
    static constexpr int BX = 32, BY = 8;              // threads
    // faces of a tile (y tiles of doubles at most 16 high: 48 KB static shared memory)
    static constexpr int FX = 32, FY = FY_;
    static constexpr int FPT = FY / BY;                // faces per thread
    static constexpr int NB = DIR == 0 ? FX : FY;      // faces per tile line
    static constexpr int NTL = DIR == 0 ? FY : FX;     // tile lines
    static constexpr int NPOS = NB + 2;                // Din positions per line
    static constexpr int NP = DIR == 0 ? NPOS : NPOS + 1;  // odd row length for y
};

// ---------------------------------------------------------------------------
// The reconstruction along a line, with every quantity computed once: Din at
// a cell from its three slopes, and from two neighbouring Din the left state
// of the face after them and the right state of the face between them.
// ---------------------------------------------------------------------------
// Din from the slopes T1 = v(p-1)-v(p-2), T2 = v(p)-v(p-1), T3 = v(p+1)-v(p)
// (ho_din): the same value as lim3's three slopes.  For slopes of one sign
// lim3(a, b, c) = s min(|a|, 2|b|, 2|c|) = s min(|a|, 2m) with m the least of
// the three sizes, else 0; so each limited slope is its own clamped to
// [2 min(0, max), 2 max(0, min)].
__device__ __forceinline__ float line_din(float T1, float T2, float T3, bool wet) {
    const float lo = 2.0f * fminf(0.0f, fmaxf(fmaxf(T1, T2), T3)), hi = 2.0f * fmaxf(0.0f, fminf(fminf(T1, T2), T3));
    const float D1 = fminf(fmaxf(T1, lo), hi), D2 = fminf(fmaxf(T2, lo), hi), D3 = fminf(fmaxf(T3, lo), hi);
    const float d = __fmaf_rn(-(1.0f / 6.0f), __fadd_rn(__fmaf_rn(-2.0f, D2, D3), D1), T2);
    return wet ? d : T2;
}
// FP64: the limiting on the bits.  A zero T2 keeps lim3's expressions, whose
// zeros' signs decide the sign of Din there (vl_guard reads it); so do
// non-finite slopes.
__device__ __forceinline__ double line_din(double T1, double T2, double T3, bool wet) {
    if (!wet) return T2;
    const unsigned long long m1 = dmag(T1), m2 = dmag(T2), m3 = dmag(T3);
    const unsigned long long mx = m1 > m2 ? (m1 > m3 ? m1 : m3) : (m2 > m3 ? m2 : m3);
    if (m2 == 0 || mx >= D_INF) {
        const double P1 = lim3(T1, T2, T3), P2 = lim3(T2, T3, T1), P3 = lim3(T3, T1, T2);
        return T2 - 1.0 / 6.0 * (P3 - 2.0 * P2 + P1);
    }
    const unsigned long long mn = m1 < m2 ? (m1 < m3 ? m1 : m3) : (m2 < m3 ? m2 : m3);
    // slopes of both signs, or a zero one: the limited slopes are zero
    if ((((dbits(T1) ^ dbits(T2)) | (dbits(T1) ^ dbits(T3))) & D_SIGN) || mn == 0) return T2;
    const unsigned long long two = (mn >> 52) ? mn + (1ull << 52) : mn << 1;  // 2 mn
    const unsigned long long sg = dbits(T2) & D_SIGN;
    const double D1 = dfrom(sg | (m1 < two ? m1 : two)), D2 = dfrom(sg | (m2 < two ? m2 : two)),
                 D3 = dfrom(sg | (m3 < two ? m3 : two));
    // D3 - 2 D2: the product is exact, so one fused operation rounds the same
    return __dsub_rn(T2, __dmul_rn(1.0 / 6.0, __dadd_rn(__fma_rn(-2.0, D2, D3), D1)));
}

// what the two pairs that a cell's Din belongs to share: in FP64 the guarded
// slope (vl_guard) and its reciprocal
template <typename T> struct LineSlope;
template <> struct LineSlope<float> {
    float t;
    __device__ __forceinline__ void set(float d) { t = d; }
};
template <> struct LineSlope<double> {
    double t, y;
    __device__ __forceinline__ void set(double d) {
        const unsigned long long m = dmag(d);
        t = m <= dbits(SMALL) ? dfrom((dbits(d) & D_SIGN) | dbits(SMALL)) : d;
        y = __drcp_rn(t);
    }
};
// vl_phi
__device__ __forceinline__ double line_phi(double rat) {
    const double s = __dadd_rn(1.0, rat);
    if (!(dbits(rat) & D_SIGN)) return __ddiv_rn(__dadd_rn(rat, rat), s);
    // rat < 0: rat + |rat| = +0 over 1 + rat, or 0 where that is small
    return ((dbits(s) & D_SIGN) && dmag(s) > dbits(SMALL) && dmag(s) <= D_INF) ? -0.0 : 0.0;
}
// the right state of the face between cells (k, k+1) is v(k) minus, the left
// state of the face after it v(k) plus, what Din of k and k+1 give (ho_lr)
__device__ __forceinline__ void line_pair(const LineSlope<float> &a, const LineSlope<float> &b, float v, float &R, float &L) {
    const float h = (a.t * b.t > 0.0f) ? __fdividef(2.0f * a.t * b.t, a.t + b.t) : 0.0f;
    R = v - 0.5f * h;
    L = v + 0.5f * h;
}
__device__ __forceinline__ void line_pair(const LineSlope<double> &a, const LineSlope<double> &b, double v, double &R, double &L) {
    double r1, r2;
    const unsigned long long big = (1023ull + 300) << 52;
    if (dmag(a.t) < big && dmag(b.t) < big) {
        // b/a and a/b by the slopes' reciprocals (their signs: Markstein's
        // steps do not depend on them)
        const double q1 = __dmul_rn(b.t, a.y), q2 = __dmul_rn(a.t, b.y);
        r1 = __fma_rn(__fma_rn(-q1, a.t, b.t), a.y, q1);
        r2 = __fma_rn(__fma_rn(-q2, b.t, a.t), b.y, q2);
    } else {
        r1 = b.t / a.t;
        r2 = a.t / b.t;
    }
    const double A = __dmul_rn(line_phi(r1), a.t), B = __dmul_rn(line_phi(r2), b.t);
    // 2 x: exact, so van * t doubled is (2 van) * t
    L = __dadd_rn(v, __dmul_rn(1.0 / 6.0, __dadd_rn(A, __dadd_rn(B, B))));
    R = __dsub_rn(v, __dmul_rn(1.0 / 6.0, __dadd_rn(__dadd_rn(A, A), B)));
}

// the three fluxes of a face (hll): in FP64 their common divisor's reciprocal
// is taken once
__device__ __forceinline__ void hll3(float SL, float SR, float F0L, float F0R, float U0L, float U0R, float F1L, float F1R,
                                     float U1L, float U1R, float F2L, float F2R, float U2L, float U2R, float &A,
                                     float &B, float &C) {
    const float r = SR - SL, d = fabsf(r) < (float)SMALL ? (float)SMALL : r, sp = SL * SR;
    const float a = SR * F0L - SL * F0R + sp * (U0R - U0L), b = SR * F1L - SL * F1R + sp * (U1R - U1L),
                c = SR * F2L - SL * F2R + sp * (U2R - U2L);
    A = SL >= 0.0f ? F0L : SR <= 0.0f ? F0R : __fdividef(a, d);
    B = SL >= 0.0f ? F1L : SR <= 0.0f ? F1R : __fdividef(b, d);
    C = SL >= 0.0f ? F2L : SR <= 0.0f ? F2R : __fdividef(c, d);
}
__device__ __forceinline__ void hll3(double SL, double SR, double F0L, double F0R, double U0L, double U0R, double F1L,
                                     double F1R, double U1L, double U1R, double F2L, double F2R, double U2L,
                                     double U2R, double &A, double &B, double &C) {
    const double ds = SR - SL;
    if (SL >= 0.0 || SR <= 0.0 || !(ds >= SMALL && ds < 0x1p300)) {
        A = hll(SL, SR, F0L, F0R, U0L, U0R);
        B = hll(SL, SR, F1L, F1R, U1L, U1R);
        C = hll(SL, SR, F2L, F2R, U2L, U2R);
        return;
    }
    const double y = __drcp_rn(ds), sp = SL * SR;
    A = div_rcp(SR * F0L - SL * F0R + sp * (U0R - U0L), ds, y);
    B = div_rcp(SR * F1L - SL * F1R + sp * (U1R - U1L), ds, y);
    C = div_rcp(SR * F2L - SL * F2R + sp * (U2R - U2L), ds, y);
}

// one face from its left and right states: wave speeds, HLL and
// BOUNDARY_CONDITION (walls and dry faces; last write wins).  pos: the face's
// index along DIR; mL, mR: MASK of the cells pos-1 and pos
template <typename T, int DIR>
__device__ __forceinline__ void face_flux(const Grid &g, const T *Lv, const T *Rv, T Dd, T m9, int pos, int mL, int mR,
                                          T &Pm, T &Nm, T &Tm) {
    const T g1 = GC(gamma1), g3 = GC(gamma3);
    const int lo = DIR == 0 ? g.ib : g.jb, hi = DIR == 0 ? g.ie : g.je;
    const T UL = Lv[0], UR = Rv[0], VL = Lv[1], VR = Rv[1], HUL = Lv[2], HUR = Rv[2];
    const T HVL = Lv[3], HVR = Rv[3], EL = Lv[4], ER = Rv[4];
    const T U4L = Lv[5], U4R = Rv[5], V4L = Lv[6], V4R = Rv[6];
    const T HL = EL + Dd, HR = ER + Dd;
    const T nL = DIR == 0 ? UL : VL, nR = DIR == 0 ? UR : VR;
    const T tL = DIR == 0 ? VL : UL, tR = DIR == 0 ? VR : UR;
    const T n4L = DIR == 0 ? U4L : V4L, n4R = DIR == 0 ? U4R : V4R;
    const T t4L = DIR == 0 ? V4L : U4L, t4R = DIR == 0 ? V4R : U4R;
    const T qnL = DIR == 0 ? HUL : HVL, qnR = DIR == 0 ? HUR : HVR;  // HU for x, HV for y
    const T qtL = DIR == 0 ? HVL : HUL, qtR = DIR == 0 ? HVR : HUR;
    // mass flux PL/QL, normal momentum flux FxL/GyL, tangential GxL/FyL
    const T ML = qnL + g1 * m9 * HL * n4L;
    const T MR = qnR + g1 * m9 * HR * n4R;
    const T NL = g3 * ML * (nL + g1 * m9 * n4L) + (T)0.5 * (T)GRAV * ((EL) * (EL)*g3 + (T)2 * (EL) * (Dd));
    const T NR = g3 * MR * (nR + g1 * m9 * n4R) + (T)0.5 * (T)GRAV * ((ER) * (ER)*g3 + (T)2 * (ER) * (Dd));
    T TL, TR;
    if (DIR == 0) {
        TL = HL * (nL + g1 * m9 * n4L) * (tL + g1 * m9 * t4L) * g3;
        TR = HR * (nR + g1 * m9 * n4R) * (tR + g1 * m9 * t4R) * g3;
    } else {
        TL = HL * (tL + g1 * m9 * t4L) * (nL + g1 * m9 * n4L) * g3;
        TR = HR * (tR + g1 * m9 * t4R) * (nR + g1 * m9 * n4R) * g3;
    }
    // WAVE_SPEED (Zhou et al. 2001)
    const T SQR_PHI_L = fsqrt((T)GRAV * fabs_(HL));
    const T SQR_PHI_R = fsqrt((T)GRAV * fabs_(HR));
    const T SQR_PHI_S = (T)0.5 * (SQR_PHI_L + SQR_PHI_R) + (T)0.25 * (nL - nR);
    const T U_S = (T)0.5 * (nL + nR) + SQR_PHI_L - SQR_PHI_R;
    const T SL = tmin(nL - SQR_PHI_L, U_S - SQR_PHI_S);
    const T SR = tmax(nR + SQR_PHI_R, U_S + SQR_PHI_S);
    hll3(SL, SR, ML, MR, EL, ER, NL, NR, qnL, qnR, TL, TR, qtL, qtR, Pm, Nm, Tm);
    // BOUNDARY_CONDITION: walls, then the dry-cell loop (last write wins)
    const bool wall_on = DIR == 0 || !g.periodic;
    if (wall_on && pos == lo) {
        Pm = (T)0;
        Nm = press(ER, Dd, g3);
        Tm = (T)0;
    }
    if (wall_on && pos == hi + 1) {
        Pm = (T)0;
        Nm = press(EL, Dd, g3);
        Tm = (T)0;
    }
    if (mL < 1) {
        Pm = (T)0;
        Nm = (pos - 1 != hi) ? press(ER, Dd, g3) * m2r<T>(mR) : (T)0;
        Tm = (T)0;
    }
    if (mR < 1) {
        Pm = (T)0;
        Nm = (pos != lo) ? press(EL, Dd, g3) * m2r<T>(mL) : (T)0;
        Tm = (T)0;
    }
}

// FLUXES along y: a thread walks `strip` faces of one column, keeping each
// field's last two cells, slopes, Din and the left state of the next face in
// registers, so that a cell is loaded once and Din, and the pair of Din that
// two faces share, are computed once.  The next face's cells are loaded while
// a face is computed (without that, 189 us at 2048 x 2048: 20 warps to an SM
// do not hide the loads).  The tiles that shared Din through shared memory
// took 790 instructions per face; this takes 400.  2048 x 2048 float: 121 ->
// 66 us (the bound: instruction issue); 701 x 937 double: 1493 -> 680 us (the
// FP64 pipe).
template <typename T>
__global__ void __launch_bounds__(128) k_flux_y(Grid g, Fields<T> f, int strip) {
    const int i = blockIdx.x * 32 + threadIdx.x;
    const int j0 = g.jb + (blockIdx.y * blockDim.y + threadIdx.y) * strip;
    if (i < g.ib || i > g.ie || j0 > g.je + 1) return;
    const int j1 = min(j0 + strip - 1, g.je + 1);
    const T *const src[7] = {f.U, f.V, f.HU, f.HV, f.Eta, f.U4, f.V4};
    const bool disp = g.dispersion != 0;
    T v1[7], v2[7], T1[7], T2[7], L[7];  // cells j-1 (then j) and j+1, their slopes, the next left state
    LineSlope<T> d[7];
    int o = i + j0 * g.pitch;
    // MASK of the cells j-3 .. j+2 of face j, bit 0 the first
    int mk = 0;
#pragma unroll
    for (int q = 0; q < 5; q++) mk |= (int)ro(f.MASK + (o + (q - 3) * g.pitch)) << q;
#pragma unroll
    for (int q = 0; q < 7; q++) {
        if (q >= 5 && !disp) {
            v1[q] = v2[q] = T1[q] = T2[q] = L[q] = (T)0;
            d[q].set((T)0);
            continue;
        }
        const T *s = src[q] + o;
        const T a = ro(s - 3 * g.pitch), b = ro(s - 2 * g.pitch), c = ro(s - g.pitch);
        v1[q] = ro(s);
        v2[q] = ro(s + g.pitch);
        const T Ta = b - a, Tb = c - b;
        T1[q] = v1[q] - c;
        T2[q] = v2[q] - v1[q];
        LineSlope<T> dm;
        dm.set(line_din(Ta, Tb, T1[q], (mk & 0xf) == 0xf));
        d[q].set(line_din(Tb, T1[q], T2[q], (mk & 0x1e) == 0x1e));
        T r;
        line_pair(dm, d[q], c, r, L[q]);
    }
    // the cells j+2 and the face's depth and masks, one face ahead
    T v3[7], Dd = ro(f.Depthy + o);
    int mq = ro(f.MASK + (o + 2 * g.pitch)), m9 = ro(f.MASK9 + o);
#pragma unroll
    for (int q = 0; q < 7; q++) v3[q] = q < 5 || disp ? ro(src[q] + (o + 2 * g.pitch)) : (T)0;
#pragma unroll 2
    for (int j = j0; j <= j1; j++, o += g.pitch) {
        mk |= mq << 5;
        const bool wet = (mk & 0x3c) == 0x3c;
        const T Dj = Dd, m9j = m2r<T>(m9);
        T c3[7];
#pragma unroll
        for (int q = 0; q < 7; q++) c3[q] = v3[q];
        if (j < j1) {
            const int on = o + g.pitch;
            Dd = ro(f.Depthy + on);
            m9 = ro(f.MASK9 + on);
            mq = ro(f.MASK + (on + 2 * g.pitch));
#pragma unroll
            for (int q = 0; q < 7; q++)
                if (q < 5 || disp) v3[q] = ro(src[q] + (on + 2 * g.pitch));
        }
        T Lv[7], Rv[7];
#pragma unroll
        for (int q = 0; q < 7; q++) {
            if (q >= 5 && !disp) {
                Lv[q] = Rv[q] = (T)0;
                continue;
            }
            const T T3 = c3[q] - v2[q];
            LineSlope<T> dn;
            dn.set(line_din(T1[q], T2[q], T3, wet));
            Lv[q] = L[q];
            line_pair(d[q], dn, v1[q], Rv[q], L[q]);
            d[q] = dn;
            v1[q] = v2[q];
            v2[q] = c3[q];
            T1[q] = T2[q];
            T2[q] = T3;
        }
        T Pm, Nm, Tm;
        face_flux<T, 1>(g, Lv, Rv, Dj, m9j, j, (mk >> 2) & 1, (mk >> 3) & 1, Pm, Nm, Tm);
        f.Q[o] = Pm;
        f.Gy[o] = Nm;
        f.Fy[o] = Tm;
        mk >>= 1;
    }
}

// FLUXES along x: a lane takes two neighbouring cells (one 8- or 16-byte load
// per field) and their two faces, and gets the neighbours' slopes, Din and
// left state from the lanes beside it; lanes 2 .. 30 have all they need, so a
// warp covers FLUX_XW = 58 faces of a row.  2048 x 2048 float: 112 -> 63 us
// (before: 32 x 8 tiles, Din through shared memory); 701 x 937 double: 1722
// -> 725 us.
constexpr int FLUX_XW = 58;
template <typename T> __device__ __forceinline__ T shup(T x) { return __shfl_up_sync(0xffffffffu, x, 1); }
template <typename T> __device__ __forceinline__ T shdn(T x) { return __shfl_down_sync(0xffffffffu, x, 1); }
__device__ __forceinline__ LineSlope<float> slope_dn(const LineSlope<float> &a) {
    LineSlope<float> r;
    r.t = shdn(a.t);
    return r;
}
__device__ __forceinline__ LineSlope<double> slope_dn(const LineSlope<double> &a) {
    LineSlope<double> r;
    r.t = shdn(a.t);
    r.y = shdn(a.y);
    return r;
}
template <typename T>
__global__ void __launch_bounds__(128) k_flux_x(Grid g, Fields<T> f, int rows) {
    using T2 = typename std::conditional<sizeof(T) == sizeof(double), double2, float2>::type;
    const int lane = threadIdx.x;
    const int i = FLUX_XW * blockIdx.x - 2 + 2 * lane;  // the lane's cells i, i+1 and the faces before them
    const int j0 = g.jb + (blockIdx.y * blockDim.y + threadIdx.y) * rows;
    if (j0 > g.je) return;
    const int j1 = min(j0 + rows - 1, g.je);
    const T *const src[7] = {f.U, f.V, f.HU, f.HV, f.Eta, f.U4, f.V4};
    const bool disp = g.dispersion != 0, mine = lane >= 2 && lane <= 30;
    // cells left of the plane's rows or past their end are other rows' cells:
    // loaded (rows 3 .. Nloc-4 of Nloc+1), never used by a face of the domain
    for (int j = j0; j <= j1; j++) {
        const int o = i + j * g.pitch;
        const uchar2 m = __ldg((const uchar2 *)(f.MASK + o));
        const int mo = (int)m.x | ((int)m.y << 1);
        // MASK of the cells i-2 .. i+3, bit 0 the first
        const int mk = shup(mo) | (mo << 2) | (shdn(mo) << 4);
        const T2 Dd = __ldg((const T2 *)(f.Depthx + o));
        const uchar2 m9 = __ldg((const uchar2 *)(f.MASK9 + o));
        T2 vv[7];
#pragma unroll
        for (int q = 0; q < 7; q++) vv[q] = q < 5 || disp ? __ldg((const T2 *)(src[q] + o)) : T2{(T)0, (T)0};
        T La[7], Ra[7], Lb[7], Rb[7];  // faces i and i+1
#pragma unroll
        for (int q = 0; q < 7; q++) {
            const T2 v = vv[q];
            const T Ta = v.x - shup(v.y), Tb = v.y - v.x;  // v(i)-v(i-1), v(i+1)-v(i)
            const T Tm = shup(Tb), Tp = shdn(Ta);
            LineSlope<T> da, db;
            da.set(line_din(Tm, Ta, Tb, (mk & 0xf) == 0xf));
            db.set(line_din(Ta, Tb, Tp, (mk & 0x1e) == 0x1e));
            T Ln;
            line_pair(da, db, v.x, Ra[q], Lb[q]);
            line_pair(db, slope_dn(da), v.y, Rb[q], Ln);
            La[q] = shup(Ln);
        }
        if (!mine) continue;
        T P0, N0, T0, P1, N1, T1;
        face_flux<T, 0>(g, La, Ra, Dd.x, m2r<T>(m9.x), i, (mk >> 1) & 1, (mk >> 2) & 1, P0, N0, T0);
        face_flux<T, 0>(g, Lb, Rb, Dd.y, m2r<T>(m9.y), i + 1, (mk >> 2) & 1, (mk >> 3) & 1, P1, N1, T1);
        if (i >= g.ib && i + 1 <= g.ie + 1) {
            *(T2 *)(f.P + o) = T2{P0, P1};
            *(T2 *)(f.Fx + o) = T2{N0, N1};
            *(T2 *)(f.Gx + o) = T2{T0, T1};
        } else if (i >= g.ib && i <= g.ie + 1) {
            f.P[o] = P0;
            f.Fx[o] = N0;
            f.Gx[o] = T0;
        } else if (i + 1 >= g.ib && i + 1 <= g.ie + 1) {
            f.P[o + 1] = P1;
            f.Fx[o + 1] = N1;
            f.Gx[o + 1] = T1;
        }
    }
}

// The tile's inputs staged by TMA: one 2-D tensor load of each of U V HU HV
// Eta U4 V4 (40 cells wide from i0 - 3, FY rows from j0 for x faces or FY+6
// rows from j0 - 3 for y faces) and of MASK (48 wide), completing on one
// mbarrier; Din of the seven fields is computed once per cell position into
// shared memory, and each thread finishes its faces from there.  i0 - 3 is a
// multiple of 32 (ib = 3), so every box starts on a 16-byte boundary.  The
// same results as k_flux_x and k_flux_y, bit for bit.
template <typename T, int DIR, int FY_> struct FluxStage {
    using TL = FluxTile<T, DIR, FY_>;
    static constexpr int BW = 40, BWM = 48;             // staged columns from i0 - 3
    static constexpr int BH = DIR == 0 ? FY_ : FY_ + 6;  // staged rows from j0 (x) or j0 - 3 (y)
    static constexpr int FB = (BW * BH * (int)sizeof(T) + 127) / 128 * 128;
    static constexpr int MB = (BWM * BH + 127) / 128 * 128;
    static constexpr int DB = (7 * TL::NTL * TL::NP * (int)sizeof(T) + 127) / 128 * 128;
    static constexpr int BYTES = 7 * FB + MB + DB + 16 + 128;
};

template <typename T> __device__ __forceinline__ T fnan();
template <> __device__ __forceinline__ float fnan<float>() { return __int_as_float(0x7fffffff); }
template <> __device__ __forceinline__ double fnan<double>() { return __longlong_as_double(0x7fffffffffffffffll); }

template <typename T, int DIR, int FY_>
__global__ void __launch_bounds__(256) k_flux_tma(Grid g, Fields<T> f, const __grid_constant__ FluxMaps maps) {
    using TL = FluxTile<T, DIR, FY_>;
    using S = FluxStage<T, DIR, FY_>;
    static_assert(TL::FY % TL::BY == 0, "whole faces per thread");
    constexpr int BX = TL::BX, BY = TL::BY, NTL = TL::NTL, NPOS = TL::NPOS, NP = TL::NP;
    extern __shared__ uint8_t fsm_raw[];
    uint8_t *sm = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(fsm_raw) + 127) & ~(uintptr_t)127);
    T(*din)[NTL][NP] = reinterpret_cast<T(*)[NTL][NP]>(sm + 7 * S::FB + S::MB);
    const uint32_t bar = fwtc::smem_u32(sm + 7 * S::FB + S::MB + S::DB);
#define FLD(v_, r_, c_) (reinterpret_cast<const T *>(sm + (v_) * S::FB)[(r_) * S::BW + (c_)])
#define MSK(r_, c_) ((int)(sm + 7 * S::FB)[(r_) * S::BWM + (c_)])
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int tid = tx + ty * BX;
    const int i0 = g.ib + blockIdx.x * TL::FX, j0 = g.jb + blockIdx.y * TL::FY;
    const int lo = DIR == 0 ? g.ib : g.jb, hi = DIR == 0 ? g.ie : g.je;
    const int base = (DIR == 0 ? i0 : j0) - 1;
    const int nvar = g.dispersion ? 7 : 5;
    if (tid == 0) {
        fwtc::mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (tid == 0) {
        const int xs = i0 - 3, ysr = DIR == 0 ? j0 : j0 - 3;
        fwtc::mbar_expect_tx(bar, (uint32_t)(nvar * S::BW * S::BH * (int)sizeof(T) + S::BWM * S::BH));
        for (int v = 0; v < nvar; v++) fwtc::tma_load_2d(fwtc::smem_u32(sm + v * S::FB), &maps.m[v], xs, ysr, bar);
        fwtc::tma_load_2d(fwtc::smem_u32(sm + 7 * S::FB), &maps.m[7], xs, ysr, bar);
    }
    const bool staged = fwtc::mbar_wait(bar, 0, maps.wait_limit ? maps.wait_limit : fwtc::WAIT_LIMIT);
    // the NTL x NPOS Din positions of the tile, spread over all threads
    for (int it = tid; it < NTL * NPOS; it += BX * BY) {
        const int k = DIR == 0 ? it % NPOS : it / NTL;
        const int ln = DIR == 0 ? it / NPOS : it % NTL;
        const int p = base + k;
        const int ci = DIR == 0 ? p : i0 + ln;
        const int cj = DIR == 0 ? j0 + ln : p;
        const bool lok = DIR == 0 ? (cj <= g.je) : (ci <= g.ie);
        if (lok && p >= lo - 1 && p <= hi + 2) {
            // cells p-2 .. p+1: staged columns k .. k+3 of row ln (x), or
            // rows k .. k+3 of column ln + 3 (y)
            int m[4];
#pragma unroll
            for (int q = 0; q < 4; q++) m[q] = DIR == 0 ? MSK(ln, k + q) : MSK(k + q, ln + 3);
#pragma unroll
            for (int vv = 0; vv < 7; vv++) {
                if (vv < nvar) {
                    T v[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) v[q] = DIR == 0 ? FLD(vv, ln, k + q) : FLD(vv, k + q, ln + 3);
                    din[vv][ln][k] = ho_din(v, m);
                }
            }
        }
    }
    __syncthreads();
    const T g1 = GC(gamma1), g3 = GC(gamma3);
    for (int r = 0; r < TL::FPT; r++) {
    const int i = i0 + tx;
    const int j = j0 + ty + r * BY;
    if (DIR == 0) {
        if (i > g.ie + 1 || j > g.je) continue;
    } else {
        if (i > g.ie || j > g.je + 1) continue;
    }
    const int own = DIR == 0 ? tx : ty + r * BY;
    const int line = DIR == 0 ? ty + r * BY : tx;
    const int fid = i + j * g.pitch;
    const int kf = own + 1;
    T Lv[7], Rv[7];
#pragma unroll
    for (int vv = 0; vv < 7; vv++) {
        if (vv >= nvar) {
            Lv[vv] = (T)0;
            Rv[vv] = (T)0;
            continue;
        }
        // cells pos-1 and pos from the staged tile
        ho_lr(FLD(vv, DIR == 0 ? line : own + 2, DIR == 0 ? own + 2 : line + 3),
              FLD(vv, DIR == 0 ? line : own + 3, DIR == 0 ? own + 3 : line + 3), din[vv][line][kf - 1],
              din[vv][line][kf], din[vv][line][kf + 1], Lv[vv], Rv[vv]);
    }
    const T UL = Lv[0], UR = Rv[0], VL = Lv[1], VR = Rv[1], HUL = Lv[2], HUR = Rv[2];
    const T HVL = Lv[3], HVR = Rv[3], EL = Lv[4], ER = Rv[4];
    const T U4L = Lv[5], U4R = Rv[5], V4L = Lv[6], V4R = Rv[6];
    const T Dd = DIR == 0 ? ro(f.Depthx + (fid)) : ro(f.Depthy + (fid));
    const T HL = EL + Dd, HR = ER + Dd;
    // MASK9u(Mloc1,:) = MASK9(Mloc,:) (fluxes.F:1333); the faces computed
    // here never reach that column
    const T m9 = m2r<T>(ro(f.MASK9 + (fid)));
    const T nL = DIR == 0 ? UL : VL, nR = DIR == 0 ? UR : VR;
    const T tL = DIR == 0 ? VL : UL, tR = DIR == 0 ? VR : UR;
    const T n4L = DIR == 0 ? U4L : V4L, n4R = DIR == 0 ? U4R : V4R;
    const T t4L = DIR == 0 ? V4L : U4L, t4R = DIR == 0 ? V4R : U4R;
    const T qnL = DIR == 0 ? HUL : HVL, qnR = DIR == 0 ? HUR : HVR;  // HU for x, HV for y
    const T qtL = DIR == 0 ? HVL : HUL, qtR = DIR == 0 ? HVR : HUR;
    // mass flux PL/QL, normal momentum flux FxL/GyL, tangential GxL/FyL
    const T ML = qnL + g1 * m9 * HL * n4L;
    const T MR = qnR + g1 * m9 * HR * n4R;
    const T NL = g3 * ML * (nL + g1 * m9 * n4L) + (T)0.5 * (T)GRAV * ((EL) * (EL)*g3 + (T)2 * (EL) * (Dd));
    const T NR = g3 * MR * (nR + g1 * m9 * n4R) + (T)0.5 * (T)GRAV * ((ER) * (ER)*g3 + (T)2 * (ER) * (Dd));
    T TL, TR;
    if (DIR == 0) {
        TL = HL * (nL + g1 * m9 * n4L) * (tL + g1 * m9 * t4L) * g3;
        TR = HR * (nR + g1 * m9 * n4R) * (tR + g1 * m9 * t4R) * g3;
    } else {
        TL = HL * (tL + g1 * m9 * t4L) * (nL + g1 * m9 * n4L) * g3;
        TR = HR * (tR + g1 * m9 * t4R) * (nR + g1 * m9 * n4R) * g3;
    }
    // WAVE_SPEED (Zhou et al. 2001)
    const T SQR_PHI_L = fsqrt((T)GRAV * fabs_(HL));
    const T SQR_PHI_R = fsqrt((T)GRAV * fabs_(HR));
    const T SQR_PHI_S = (T)0.5 * (SQR_PHI_L + SQR_PHI_R) + (T)0.25 * (nL - nR);
    const T U_S = (T)0.5 * (nL + nR) + SQR_PHI_L - SQR_PHI_R;
    const T SL = tmin(nL - SQR_PHI_L, U_S - SQR_PHI_S);
    const T SR = tmax(nR + SQR_PHI_R, U_S + SQR_PHI_S);
    T Pm = hll(SL, SR, ML, MR, EL, ER);
    T Nm = hll(SL, SR, NL, NR, qnL, qnR);
    T Tm = hll(SL, SR, TL, TR, qtL, qtR);
    // BOUNDARY_CONDITION: walls, then the dry-cell loop (last write wins)
    const int pos = DIR == 0 ? i : j;
    const bool wall_on = DIR == 0 || !g.periodic;
    if (wall_on && pos == lo) {
        Pm = (T)0;
        Nm = press(ER, Dd, g3);
        Tm = (T)0;
    }
    if (wall_on && pos == hi + 1) {
        Pm = (T)0;
        Nm = press(EL, Dd, g3);
        Tm = (T)0;
    }
    const int mL = MSK(DIR == 0 ? line : own + 2, DIR == 0 ? own + 2 : line + 3);  // cell pos-1
    const int mR = MSK(DIR == 0 ? line : own + 3, DIR == 0 ? own + 3 : line + 3);  // cell pos
    if (mL < 1) {
        Pm = (T)0;
        Nm = (pos - 1 != hi) ? press(ER, Dd, g3) * m2r<T>(mR) : (T)0;
        Tm = (T)0;
    }
    if (mR < 1) {
        Pm = (T)0;
        Nm = (pos != lo) ? press(EL, Dd, g3) * m2r<T>(mL) : (T)0;
        Tm = (T)0;
    }
    if (!staged) {  // the tile never arrived: poison the fluxes (the step reports NaN)
        Pm = Nm = Tm = fnan<T>();
    }
    if (DIR == 0) {
        f.P[fid] = Pm;
        f.Fx[fid] = Nm;
        f.Gx[fid] = Tm;
    } else {
        f.Q[fid] = Pm;
        f.Gy[fid] = Nm;
        f.Fy[fid] = Tm;
    }
    }
    // the tile never arrived: its copies may still be in flight; one more
    // bounded wait (the full limit) keeps this block's shared memory until
    // they land
    if (!staged && tid == 0) fwtc::mbar_wait(bar, 0, fwtc::WAIT_LIMIT);
}

#undef FLD
#undef MSK

// ---------------------------------------------------------------------------
// SourceTerms (sources.F:56-548) at one interior cell, with the wavemaker
// mass of WK_REG / JON_2D (sources.F:109-134).
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ T wavemaker_mass(const Grid &g, const Fields<T> &f, int i, int j, double TIME) {
    if (i < g.ilo || i > g.ihi || j < g.jlo || j > g.jhi) return (T)0;
    if constexpr (sizeof(T) == sizeof(double)) {
        if (g.wavemaker == FW_WK_REG) {
            const T AA = ftanh((T)PI_SP / ((T)g.time_ramp * (T)g.tperiod) * (T)TIME) * (T)g.D_gen;
            const T xmk = (T)(i - g.ib) * (T)g.DX, ymk = (T)(j - g.jb) * (T)g.DY;
            const T dxm = xmk - (T)g.xc_wk;
            return AA * fexp(-(T)g.beta_gen * (dxm * dxm)) *
                   fsin((T)g.rlamda * (ymk - (T)0) - (T)2 * (T)PI_SP / (T)g.tperiod * (T)TIME);
        }
        if (g.wavemaker == FW_WK_JON_2D) {
            const T AA = ftanh((T)PI_SP / ((T)g.time_ramp / (T)g.freq_peak) * (T)TIME);
            const int bw = g.ihi - g.ilo + 1, bh = g.jhi - g.jlo + 1;
            const size_t b = (size_t)(i - g.ilo) + (size_t)(j - g.jlo) * bw;
            T s = (T)0;
            for (int k = 0; k < g.nfreq; k++)
                s = s + AA * ((T)f.Cm[b + (size_t)k * bw * bh] * (T)f.wmcs[2 * k] +
                              (T)f.Sm[b + (size_t)k * bw * bh] * (T)f.wmcs[2 * k + 1]);
            return s;
        }
    } else {
        // mixed: the ramp and phase of this step come from k_dt_final
        const T AA = f.fsc[FS_WKAA];
        if (g.wavemaker == FW_WK_REG) {
            const T xmk = i2r<T>(i - g.ib) * g.f_DX, ymk = i2r<T>(j - g.jb) * g.f_DY;
            const T dxm = xmk - g.f_xc_wk;
            return AA * fexp(-g.f_beta_gen * (dxm * dxm)) * fsin(g.f_rlamda * ymk - f.fsc[FS_WKPH]);
        }
        if (g.wavemaker == FW_WK_JON_2D) {
            const int bw = g.ihi - g.ilo + 1, bh = g.jhi - g.jlo + 1;
            const size_t b = (size_t)(i - g.ilo) + (size_t)(j - g.jlo) * bw;
            T s = (T)0;
            for (int k = 0; k < g.nfreq; k++)
                s = s + AA * ((T)f.Cm[b + (size_t)k * bw * bh] * f.wmcsf[2 * k] +
                              (T)f.Sm[b + (size_t)k * bw * bh] * f.wmcsf[2 * k + 1]);
            return s;
        }
    }
    return (T)0;
}

// The JON_2D mass depends on TIME, which stays through a step's three stages: a
// whole step sums the band's frequencies once, beside the first stage's
// dispersion, into the words behind Cm.  Summed in every stage's k_update, the
// warps of the band kept the others waiting (k_update at 2048 x 2048 128 ->
// 110 us, 1024 x 1024 50 -> 37).  The words are zero until a first whole step.
template <typename T> __host__ __device__ __forceinline__ T *wm_band(const Grid &g, const Fields<T> &f) {
    return f.Cm + (size_t)g.nfreq * (size_t)(g.ihi - g.ilo + 1) * (size_t)(g.jhi - g.jlo + 1);
}
template <typename T> __global__ void __launch_bounds__(256) k_wm_band(Grid g, Fields<T> f) {
    const int bw = g.ihi - g.ilo + 1, n = bw * (g.jhi - g.jlo + 1);
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= n) return;
    const int j = b / bw, i = b - j * bw;
    wm_band(g, f)[b] = wavemaker_mass(g, f, g.ilo + i, g.jlo + j, f.dsc[S_TIME]);
}

// SourceTerms at one cell; BX, BY get BreakSourceX/Y (sources.F:428-456),
// zero without viscosity breaking
template <typename T>
__device__ __forceinline__ void source_terms_b(const Grid &g, const Fields<T> &f, int i, int j, T wm, T &SX,
                                               T &SY, T &BX, T &BY) {
    BX = (T)0;
    BY = (T)0;
    constexpr bool EXACT = sizeof(T) == sizeof(double);
    const T DX = GC(DX), DY = GC(DY), mdf = GC(min_depth_frc);
    const T rdx = GC(rdx), rdy = GC(rdy);
    // x/DX: the reference's division in FP64, a reciprocal in the mixed path
#define OX(x) over((x), DX, rdx)
#define OY(x) over((x), DY, rdy)
    const T g1 = GC(gamma1), g2 = GC(gamma2);
    const size_t id = IDX(i, j);
    const size_t ie_ = IDX(i + 1, j), iw = IDX(i - 1, j), in_ = IDX(i, j + 1), is = IDX(i, j - 1);
    const T U = ro(f.U + (id)), V = ro(f.V + (id));
    const T spd = fsqrt(U * U + V * V);
    const T m9 = m2r<T>(ro(f.MASK9 + (id)));
    const T mk = m2r<T>(ro(f.MASK + (id)));
    const T Hm = tmax(f.H[id], mdf);
    const T Eta = f.Eta[id];
    const T U4 = ro(f.U4 + (id)), V4 = ro(f.V4 + (id));
    const T dPQ = OX(ro(f.P + (ie_)) - ro(f.P + (id))) + OY(ro(f.Q + (in_)) - ro(f.Q + (id)));
    const T FrcInsX = -ro(f.Cd + (id)) * U * spd;
    T sx = OX((T)GRAV * (Eta)) * (ro(f.Depthx + (ie_)) - ro(f.Depthx + (id))) * mk + FrcInsX +
           g1 * m9 * Hm *
               (OX(U * (T)0.5 * (ro(f.U4 + (ie_)) - ro(f.U4 + (iw)))) + OY(V * (T)0.5 * (ro(f.U4 + (in_)) - ro(f.U4 + (is)))) +
                OX(U4 * (T)0.5 * (ro(f.U + (ie_)) - ro(f.U + (iw)))) + OY(V4 * (T)0.5 * (ro(f.U + (in_)) - ro(f.U + (is)))) -
                g2 * m9 * ro(f.Udisp + (id))) +
           g1 * m9 * dPQ * (U4 - ro(f.U1p + (id))) + wm * U;
    const T FrcInsY = -ro(f.Cd + (id)) * V * spd;
    T sy = OY((T)GRAV * (Eta)) * (ro(f.Depthy + (in_)) - ro(f.Depthy + (id))) * mk + FrcInsY +
           g1 * m9 * Hm *
               (OX(U * (T)0.5 * (ro(f.V4 + (ie_)) - ro(f.V4 + (iw)))) + OY(V * (T)0.5 * (ro(f.V4 + (in_)) - ro(f.V4 + (is)))) +
                OX(U4 * (T)0.5 * (ro(f.V + (ie_)) - ro(f.V + (iw)))) + OY(V4 * (T)0.5 * (ro(f.V + (in_)) - ro(f.V + (is)))) -
                g2 * m9 * ro(f.Vdisp + (id))) +
           g1 * m9 * dPQ * (V4 - ro(f.V1p + (id))) + wm * V;
    if (g.friction_sponge) {
        sx = sx - ro(f.CD4 + (id)) * U * spd * ro(f.Depth + (id));
        sy = sy - ro(f.CD4 + (id)) * V * spd * ro(f.Depth + (id));
    }
    if (g.visc_breaking) {
        // nu_vis is a float array (sources.F:69): the face sums are float sums
        const float nc = (float)ro(f.nu + (id));
        const T nxp = (T)((float)ro(f.nu + (ie_)) + nc), nxm = (T)((float)ro(f.nu + (iw)) + nc);
        const T nyp = (T)((float)ro(f.nu + (in_)) + nc), nym = (T)((float)ro(f.nu + (is)) + nc);
        const T HUc = ro(f.HU + (id)), HVc = ro(f.HV + (id));
        T bx, by;
        if constexpr (EXACT) {
            // 0.5 / DX = half of RN(1/DX)
            const T hx = (T)0.5 * rdx, hy = (T)0.5 * rdy;
            const T qxp = OX(nxp), qxm = OX(nxm), qyp = OY(nyp), qym = OY(nym);
            bx = hx * (qxp * (ro(f.HU + (ie_)) - HUc) - qxm * (HUc - ro(f.HU + (iw)))) +
                 hy * (qyp * (ro(f.HU + (in_)) - HUc) - qym * (HUc - ro(f.HU + (is))));
            by = hx * (qxp * (ro(f.HV + (ie_)) - HVc) - qxm * (HVc - ro(f.HV + (iw)))) +
                 hy * (qyp * (ro(f.HV + (in_)) - HVc) - qym * (HVc - ro(f.HV + (is))));
        } else {
            const T cx = (T)g.f_cx, cy = (T)g.f_cy;
            bx = cx * (nxp * (ro(f.HU + (ie_)) - HUc) - nxm * (HUc - ro(f.HU + (iw)))) +
                 cy * (nyp * (ro(f.HU + (in_)) - HUc) - nym * (HUc - ro(f.HU + (is))));
            by = cx * (nxp * (ro(f.HV + (ie_)) - HVc) - nxm * (HVc - ro(f.HV + (iw)))) +
                 cy * (nyp * (ro(f.HV + (in_)) - HVc) - nym * (HVc - ro(f.HV + (is))));
        }
        sx = sx + bx;
        sy = sy + by;
        BX = bx;
        BY = by;
    }
#undef OX
#undef OY
    SX = sx;
    SY = sy;
}
template <typename T>
__device__ __forceinline__ void source_terms(const Grid &g, const Fields<T> &f, int i, int j, T wm, T &SX,
                                             T &SY) {
    T bx, by;
    source_terms_b(g, f, i, j, wm, SX, SY, bx, by);
}

// SourceTerms alone (materialises SourceX, SourceY, WaveMaker_Mass)
template <typename T>
__global__ void __launch_bounds__(256) k_sources(Grid g, Fields<T> f) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x + g.ib;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + g.jb;
    if (i > g.ie || j > g.je) return;
    const T wm = wavemaker_mass(g, f, i, j, f.dsc[S_TIME]);
    T sx, sy;
    source_terms(g, f, i, j, wm, sx, sy);
    f.SourceX[IDX(i, j)] = sx;
    f.SourceY[IDX(i, j)] = sy;
    f.WM[IDX(i, j)] = wm;
}

// ---------------------------------------------------------------------------
// ESTIMATE_HUV (etauv_solver.F:53-351) fused with SourceTerms, plus the H
// update and the right-hand sides of the tridiagonal systems of
// GET_Eta_U_V_HU_HV (etauv_solver.F:365-539).  RAD (the last two stages,
// with the radiation sums on) also stores P_center, Q_center, U_davg, V_davg
// with the stage's starting H (etauv_solver.F:94-101), Wsurf = R1
// (etauv_solver.F:247) and BreakSourceX/Y.  BAND: the wavemaker's mass comes from
// k_wm_band.
// ---------------------------------------------------------------------------
template <typename T, bool RAD, bool BAND>
__global__ void __launch_bounds__(256, sizeof(T) == sizeof(float) ? 4 : 3) k_update(Grid g, Fields<T> f, T al, T be, Ahead ah) {
    prefetch_ahead<T>(g, ah, blockIdx.y, 0);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= g.Mloc || j >= g.Nloc) return;
    const size_t id = IDX(i, j);
    const T g3 = GC(gamma3);
    if (i < g.ib || i > g.ie || j < g.jb || j > g.je) {
        f.H[id] = f.Eta[id] * g3 + ro(f.Depth + (id));  // H = Eta*Gamma3+Depth on all cells
        return;
    }
    if constexpr (sizeof(T) == sizeof(float)) {
        // the right-hand sides' inputs (rows j-1..j+1 of U, V, Depth, the
        // masks), read after this kernel's stores
        if (g.dispersion) {
#pragma unroll
            for (int b = -1; b <= 1; b++) {
                prefetch_l1(f.U + IDX(i, j + b));
                prefetch_l1(f.V + IDX(i, j + b));
                prefetch_l1(f.Depth + IDX(i, j + b));
            }
            prefetch_l1(f.MASK9 + id);
            prefetch_l1(f.MASK + id);
        }
    }
    const T DX = GC(DX), DY = GC(DY);
    const T DT = DTV;
    T wm = (T)0;
    if constexpr (BAND) {
        if (i >= g.ilo && i <= g.ihi && j >= g.jlo && j <= g.jhi)
            wm = ro(wm_band(g, f) + (i - g.ilo) + (j - g.jlo) * (g.ihi - g.ilo + 1));
    } else {
        wm = wavemaker_mass(g, f, i, j, f.dsc[S_TIME]);
    }
    T SX, SY, BX, BY;
    source_terms_b(g, f, i, j, wm, SX, SY, BX, BY);

    const size_t ie_ = IDX(i + 1, j), in_ = IDX(i, j + 1);
    constexpr bool EXACT = sizeof(T) == sizeof(double);
    const T cdx = GC(rdx), cdy = GC(rdy);
    T R1 = -cdx * (ro(f.P + (ie_)) * (T)1 + ro(f.P + (id)) * (T)-1) - cdy * (ro(f.Q + (in_)) * (T)1 + ro(f.Q + (id)) * (T)-1);
    if (g.wavemaker != FW_WK_NONE) {
        const T xmk = i2r<T>(i - g.ib) * DX, ymk = i2r<T>(j - g.jb) * DY;
        if (fabs_(xmk - GC(xc_wk)) < GC(width_wk) && fabs_(ymk - GC(yc_wk)) < GC(ywidth_wk) / (T)2)
            R1 = R1 + wm;
    }
    if constexpr (RAD) {
        const size_t PL = (size_t)g.pitch * (size_t)(g.Nloc + 1);
        const T pc = (T)0.5 * (ro(f.P + (ie_)) + ro(f.P + (id))), qc = (T)0.5 * (ro(f.Q + (in_)) + ro(f.Q + (id)));
        const T hm = tmax(f.H[id], GC(min_depth_frc));  // H before this stage's update
        f.rad[RP_PC * PL + id] = pc;
        f.rad[RP_QC * PL + id] = qc;
        f.rad[RP_UD * PL + id] = pc / hm;
        f.rad[RP_VD * PL + id] = qc / hm;
        f.rad[RP_WS * PL + id] = R1;
        f.rad[RP_BX * PL + id] = BX;
        f.rad[RP_BY * PL + id] = BY;
    }
    T eta = al * ro(f.Eta0 + (id)) + be * (f.Eta[id] + DT * R1);
    if (g.eta_limiter) {
        if (eta < GC(trough)) eta = GC(trough);
        if (eta > GC(crest)) eta = GC(crest);
    }
    const T R2 = -cdx * (ro(f.Fx + (ie_)) * (T)1 + ro(f.Fx + (id)) * (T)-1) - cdy * (ro(f.Fy + (in_)) * (T)1 + ro(f.Fy + (id)) * (T)-1) + SX;
    const T ubar = al * ro(f.Ubar0 + (id)) + be * (f.Ubar[id] + DT * R2);
    const T R3 = -cdx * (ro(f.Gx + (ie_)) * (T)1 + ro(f.Gx + (id)) * (T)-1) - cdy * (ro(f.Gy + (in_)) * (T)1 + ro(f.Gy + (id)) * (T)-1) + SY;
    const T vbar = al * ro(f.Vbar0 + (id)) + be * (f.Vbar[id] + DT * R3);
    f.Eta[id] = eta;
    f.Ubar[id] = ubar;
    f.Vbar[id] = vbar;
    const T H = eta * g3 + ro(f.Depth + (id));
    f.H[id] = H;
    if (!g.dispersion) return;

    // tmp4 of the x and y systems (etauv_solver.F:410-411, 508-509)
    if constexpr (sizeof(T) == sizeof(double)) {
        const double mdf = g.min_depth_frc;
        const double g1 = g.gamma1, b1 = g.b1, b2 = g.b2;
        const double m9 = (double)ro(f.MASK9 + (id));
        const double mk = (double)ro(f.MASK + (id));
        const double dep = tmax((double)ro(f.Depth + (id)), mdf);
        const double Hm = tmax((double)H, mdf);
        // the cross derivatives CAL_DISPERSION left at the start of the stage
        const double Vxy = ro(f.Vxy + (id)), DVxy = ro(f.DVxy + (id)), Uxy = ro(f.Uxy + (id)), DUxy = ro(f.DUxy + (id));
        const double rH = __drcp_rn(Hm);
        f.rhs_x[id] = div_any((double)ubar * mk, Hm, rH) + g1 * m9 * (-b1 / 2.0 * dep * dep * Vxy - b2 * dep * DVxy);
        f.rhs_y[id] = div_any((double)vbar * mk, Hm, rH) + g1 * m9 * (-b1 / 2.0 * dep * dep * Uxy - b2 * dep * DUxy);
    } else {
        // mixed: float arithmetic; the cross derivatives of the stage-start
        // U, V are recomputed here
        const T mf = g.f_min_depth_frc;
        const T m9 = m2r<T>(ro(f.MASK9 + (id))), mk = m2r<T>(ro(f.MASK + (id)));
        const T dep = tmax(ro(f.Depth + (id)), mf);
        const bool wall = (i == g.ib) || (i == g.ie) || (j == g.jb) || (j == g.je);
        T Vxy = (T)0, DVxy = (T)0, Uxy = (T)0, DUxy = (T)0;
        if (!wall) {
            const T q = g.f_rdxy4 * m9;
#define XY(F) (((F(1, 1) - F(1, -1)) - (F(-1, 1) - F(-1, -1))) * q)
#define LV(a, b) (ro(f.V + (IDX(i + (a), j + (b)))))
#define LU(a, b) (ro(f.U + (IDX(i + (a), j + (b)))))
#define LDV(a, b) (tmax(ro(f.Depth + (IDX(i + (a), j + (b)))), mf) * LV(a, b))
#define LDU(a, b) (tmax(ro(f.Depth + (IDX(i + (a), j + (b)))), mf) * LU(a, b))
            Vxy = XY(LV);
            DVxy = XY(LDV);
            Uxy = XY(LU);
            DUxy = XY(LDU);
#undef XY
#undef LV
#undef LU
#undef LDV
#undef LDU
        }
        const T fg = g.f_gamma1 * m9, rH = (T)1 / tmax(H, mf);
        f.rhs_x[id] = ubar * mk * rH + fg * (g.f_hb1 * dep * dep * Vxy - g.f_b2 * dep * DVxy);
        f.rhs_y[id] = vbar * mk * rH + fg * (g.f_hb1 * dep * dep * Uxy - g.f_b2 * dep * DUxy);
    }
}

// ---------------------------------------------------------------------------
// Tridiagonal u/v recovery (TRIDx_ser / TRIDy_ser / TRIDy_periodic,
// tridiagnal.F:59-398) as a partitioned line solver in double:
//   A: every chunk of m rows eliminates its interior rows for three right-
//      hand sides and emits two rows of a reduced tridiagonal system;
//   B: one thread per line solves the reduced system (two right-hand sides
//      and the Sherman-Morrison combination for periodic y);
//   C: every chunk back-substitutes its interior rows.
// Rows are the reference's normalised rows a x(k-1) + x(k) + c x(k+1) = d.
// ---------------------------------------------------------------------------
template <typename T, int DIR>
__device__ __forceinline__ void tri_coef(const Grid &g, const Fields<T> &f, int i, int j, double &a, double &c,
                                         double &d) {
    const double mdf = g.min_depth_frc, g1 = g.gamma1;
    const size_t id = IDX(i, j);
    const double dep = tmax((double)f.Depth[id], mdf);
    const double depl = tmax((double)f.Depth[DIR == 0 ? IDX(i - 1, j) : IDX(i, j - 1)], mdf);
    const double depr = tmax((double)f.Depth[DIR == 0 ? IDX(i + 1, j) : IDX(i, j + 1)], mdf);
    const double m9 = (double)f.MASK9[id];
    const double tmp4 = DIR == 0 ? f.rhs_x[id] : f.rhs_y[id];
    double tmp1, tmp2, tmp3;
    if constexpr (sizeof(T) == sizeof(double)) {
        // the reference's expressions (etauv_solver.F:406-409, 504-507);
        // their constant left parts (b1 / 2.0 / h / h and so on) come
        // evaluated in the same order
        const double k1 = g.tK1[DIR], k2 = g.tK2[DIR], k3 = g.tK3[DIR], k4 = g.tK4[DIR];
        tmp1 = g1 * m9 * (k1 * dep * dep + k2 * depl * dep);
        tmp2 = 1.0 + g1 * m9 * (k3 * dep * dep - k4 * dep * dep);
        tmp3 = g1 * m9 * (k1 * dep * dep + k2 * dep * depr);
        if (tmp2 != 0.0 || f.MASK[id] > 0) {
            a = tmp1 / tmp2;
            c = tmp3 / tmp2;
            d = tmp4 / tmp2;
        } else {
            a = 0.0;
            c = 0.0;
            d = 0.0;
        }
    } else {
        // mixed: the same coefficients from per-direction constants and one
        // reciprocal
        const double gm = g1 * m9;
        tmp1 = gm * dep * (g.cA[DIR] * dep + g.cB[DIR] * depl);
        tmp2 = 1.0 + gm * g.cC[DIR] * dep * dep;
        tmp3 = gm * dep * (g.cA[DIR] * dep + g.cB[DIR] * depr);
        if (tmp2 != 0.0 || f.MASK[id] > 0) {
            const double r = 1.0 / tmp2;
            a = tmp1 * r;
            c = tmp3 * r;
            d = tmp4 * r;
        } else {
            a = 0.0;
            c = 0.0;
            d = 0.0;
        }
    }
}

// row k (0..L-1) of line l -> cell
template <int DIR> __device__ __forceinline__ void line_cell(const Grid &g, int l, int k, int &i, int &j) {
    if (DIR == 0) {
        i = g.ib + k;
        j = g.jb + l;
    } else {
        i = g.ib + l;
        j = g.jb + k;
    }
}

// coefficients of row k of line l, with the periodic end-row scaling of
// TRIDy_periodic (tridiagnal.F:168-173) when PER
template <typename T, int DIR, bool PER>
__device__ __forceinline__ void row_coef(const Grid &g, const Fields<T> &f, const LinePart &lp, int l, int k,
                                         double &a, double &c, double &d) {
    int i, j;
    line_cell<DIR>(g, l, k, i, j);
    tri_coef<T, DIR>(g, f, i, j, a, c, d);
    if (PER) {
        if (k == 0) {
            double a2, c2, d2;
            int ie2, je2;
            line_cell<DIR>(g, l, lp.L - 1, ie2, je2);
            tri_coef<T, DIR>(g, f, ie2, je2, a2, c2, d2);  // c_end
            c = c / (1 + c2);
            d = d / (1 + c2);
        } else if (k == lp.L - 1) {
            double a2, c2, d2;
            int ib2, jb2;
            line_cell<DIR>(g, l, 0, ib2, jb2);
            tri_coef<T, DIR>(g, f, ib2, jb2, a2, c2, d2);  // a_beg
            a = a / (1 + a2);
            d = d / (1 + a2);
        }
    }
}

template <int DIR>
__device__ __forceinline__ void chunk_of(const LinePart &lp, int t, int &l, int &ch) {
    // x lines: consecutive threads walk the chunks of one line;
    // y lines: consecutive threads walk neighbouring lines (coalesced)
    if (DIR == 0) {
        l = t / lp.P;
        ch = t % lp.P;
    } else {
        ch = t / lp.nlines;
        l = t % lp.nlines;
    }
}

template <typename T, int DIR, bool PER>
__global__ void __launch_bounds__(128) k_tri_a(Grid g, Fields<T> f, LinePart lp) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= lp.nlines * lp.P) return;
    int l, ch;
    chunk_of<DIR>(lp, t, l, ch);
    const int s = ch * lp.m;
    const int e = (ch == lp.P - 1) ? lp.L - 1 : s + lp.m - 1;
    double as, cs, ds, ae, ce, de;
    row_coef<T, DIR, PER>(g, f, lp, l, s, as, cs, ds);
    row_coef<T, DIR, PER>(g, f, lp, l, e, ae, ce, de);
    if (s == 0) as = 0.0;           // first row: no lower neighbour
    if (e == lp.L - 1) ce = 0.0;    // last row: no upper neighbour
    double lo_s, di_s, up_s, r_s, lo_e, di_e, up_e, r_e;
    if (e - s >= 2) {
        // interior rows s+1..e-1: forward sweep with three right-hand sides
        double cp = 0.0, yp = 0.0, pp = 0.0, qp = 0.0;
        for (int k = s + 1; k <= e - 1; k++) {
            double a, c, d;
            row_coef<T, DIR, PER>(g, f, lp, l, k, a, c, d);
            const double lower = (k > s + 1) ? a : 0.0;
            const double r = 1.0 / (1.0 - lower * cp);
            const double upper = (k < e - 1) ? c : 0.0;
            cp = upper * r;
            yp = (d - lower * yp) * r;
            pp = ((k == s + 1 ? a : 0.0) - lower * pp) * r;
            qp = ((k == e - 1 ? c : 0.0) - lower * qp) * r;
            int ii, jj;
            line_cell<DIR>(g, l, k, ii, jj);
            const size_t q = IDX(ii, jj);
            f.ty[q] = yp;
            f.tp[q] = pp;
            f.tq[q] = qp;
            f.tc[q] = cp;  // c' for the backward sweep
        }
        // backward sweep
        double yn = 0.0, pn = 0.0, qn = 0.0;
        double y1 = 0, p1 = 0, q1 = 0, yl = 0, pl = 0, ql = 0;
        for (int k = e - 1; k >= s + 1; k--) {
            int ii, jj;
            line_cell<DIR>(g, l, k, ii, jj);
            const size_t q = IDX(ii, jj);
            const double cpk = f.tc[q];
            const double yk = f.ty[q] - cpk * yn;
            const double pk = f.tp[q] - cpk * pn;
            const double qk = f.tq[q] - cpk * qn;
            f.ty[q] = yk;
            f.tp[q] = pk;
            f.tq[q] = qk;
            yn = yk;
            pn = pk;
            qn = qk;
            if (k == e - 1) {
                yl = yk;
                pl = pk;
                ql = qk;
            }
            if (k == s + 1) {
                y1 = yk;
                p1 = pk;
                q1 = qk;
            }
        }
        lo_s = as;
        di_s = 1.0 - cs * p1;
        up_s = -cs * q1;
        r_s = ds - cs * y1;
        lo_e = -ae * pl;
        di_e = 1.0 - ae * ql;
        up_e = ce;
        r_e = de - ae * yl;
    } else {
        lo_s = as;
        di_s = 1.0;
        up_s = cs;
        r_s = ds;
        lo_e = ae;
        di_e = 1.0;
        up_e = ce;
        r_e = de;
    }
    double *red = f.red + ((size_t)l * 2 * lp.P + 2 * ch) * 6;
    red[0] = lo_s;
    red[1] = di_s;
    red[2] = up_s;
    red[3] = r_s;
    red[4] = (PER && s == 0) ? 1.0 : 0.0;  // second right-hand side (scaled below)
    red[6 + 0] = lo_e;
    red[6 + 1] = di_e;
    red[6 + 2] = up_e;
    red[6 + 3] = r_e;
    red[6 + 4] = (PER && e == lp.L - 1) ? 1.0 : 0.0;
}

template <typename T, int DIR, bool PER>
__global__ void __launch_bounds__(128) k_tri_b(Grid g, Fields<T> f, LinePart lp) {
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= lp.nlines) return;
    const int n = 2 * lp.P;
    double *red = f.red + (size_t)l * n * 6;
    double a_beg = 0.0, c_end = 0.0;
    if (PER) {
        double a, c, d;
        int i, j;
        line_cell<DIR>(g, l, 0, i, j);
        tri_coef<T, DIR>(g, f, i, j, a, c, d);
        a_beg = a;
        line_cell<DIR>(g, l, lp.L - 1, i, j);
        tri_coef<T, DIR>(g, f, i, j, a, c, d);
        c_end = c;
        // e = [1/(1+c_end), 0, ..., 0, -1/(1+a_beg)] (tridiagnal.F:207-215)
        red[4] = 1.0 / (1.0 + c_end);
        red[(size_t)(n - 1) * 6 + 4] = -1.0 / (1.0 + a_beg);
    }
    // Thomas on the reduced rows: slot 5 keeps c', slots 3/4 the rhs
    double cp = 0.0, r1 = 0.0, r2 = 0.0;
    for (int k = 0; k < n; k++) {
        double *row = red + (size_t)k * 6;
        const double lo = (k > 0) ? row[0] : 0.0;
        const double den = row[1] - lo * cp;
        cp = (k < n - 1 ? row[2] : 0.0) / den;
        r1 = (row[3] - lo * r1) / den;
        row[5] = cp;
        row[3] = r1;
        if (PER) {
            r2 = (row[4] - lo * r2) / den;
            row[4] = r2;
        }
    }
    double x1 = 0.0, x2 = 0.0;
    for (int k = n - 1; k >= 0; k--) {
        double *row = red + (size_t)k * 6;
        x1 = row[3] - row[5] * x1;
        row[3] = x1;
        if (PER) {
            x2 = row[4] - row[5] * x2;
            row[4] = x2;
        }
    }
    if (PER) {
        const double y1b = red[3], y1e = red[(size_t)(n - 1) * 6 + 3];
        const double y2b = red[4], y2e = red[(size_t)(n - 1) * 6 + 4];
        const double beta = (c_end * y1b - a_beg * y1e) / (1.0 - (c_end * y2b - a_beg * y2e));
        for (int k = 0; k < n; k++) {
            double *row = red + (size_t)k * 6;
            row[3] = row[3] + beta * row[4];
        }
    }
}

template <typename T, int DIR>
__global__ void __launch_bounds__(128) k_tri_c(Grid g, Fields<T> f, LinePart lp) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= lp.nlines * lp.P) return;
    int l, ch;
    chunk_of<DIR>(lp, t, l, ch);
    const int s = ch * lp.m;
    const int e = (ch == lp.P - 1) ? lp.L - 1 : s + lp.m - 1;
    const double *red = f.red + ((size_t)l * 2 * lp.P + 2 * ch) * 6;
    const double xs = red[3], xe = red[6 + 3];
    T *out = DIR == 0 ? f.U : f.V;
    int i, j;
    line_cell<DIR>(g, l, s, i, j);
    out[IDX(i, j)] = (T)xs;
    line_cell<DIR>(g, l, e, i, j);
    out[IDX(i, j)] = (T)xe;
    for (int k = s + 1; k <= e - 1; k++) {
        line_cell<DIR>(g, l, k, i, j);
        const size_t q = IDX(i, j);
        out[q] = (T)(f.ty[q] - f.tp[q] * xs - f.tq[q] * xe);
    }
}

// FP64: the reference's Thomas recurrence (TRIDx_ser / TRIDy_ser,
// tridiagnal.F:338-398; periodic y: TRIDy_periodic, :59-325) in its own
// operation order, in two kernels.
//   k_thomas_rows (one thread per cell) computes every row's a, c, d
//   (etauv_solver.F:406-409, 504-507), with TRIDy_periodic's end-row
//   scaling, and stores what the recurrence needs: 1/a, c/a, d/a for a row
//   that is eliminated (a != 0 and not the first row), else 0, c, d.
//   k_thomas_lines (one thread per line) then walks the line: only the
//   dependent part, den = 1/a - c'(k-1), c' = (c/a)/den and
//   d' = (d/a - d'(k-1))/den, is on its critical path, and the loads of the
//   next block of rows are issued before the current block is worked.
// The results equal the one-pass recurrence bit for bit: the same IEEE
// operations on the same operands, in a translation unit compiled without
// contraction.  Scratch: tc = 1/a, tp = c/a then c', ty = d/a then d' then
// the first solution, tq = e' then the second solution (periodic).
template <typename T, int DIR, bool PER>
__global__ void __launch_bounds__(256) k_thomas_rows(Grid g, Fields<T> f, LinePart lp) {
    const int i = g.ib + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = g.jb + blockIdx.y * blockDim.y + threadIdx.y;
    if (i > g.ie || j > g.je) return;
    const int k = DIR == 0 ? i - g.ib : j - g.jb;
    double a, c, d;
    tri_coef<T, DIR>(g, f, i, j, a, c, d);
    if (PER) {
        if (k == 0) {  // scaled by 1 + c_end, the c of the line's last row
            double a2, c2, d2;
            tri_coef<T, DIR>(g, f, DIR == 0 ? g.ie : i, DIR == 0 ? j : g.je, a2, c2, d2);
            c = c / (1 + c2);
            d = d / (1 + c2);
        }
        if (k == lp.L - 1) {  // scaled by 1 + a_beg, the a of the first row
            double a2, c2, d2;
            tri_coef<T, DIR>(g, f, DIR == 0 ? g.ib : i, DIR == 0 ? j : g.jb, a2, c2, d2);
            a = a / (1 + a2);
            d = d / (1 + a2);
        }
    }
    const size_t q = IDX(i, j);
    if (k > 0 && a != 0.0) {
        f.tc[q] = 1.0 / a;
        f.tp[q] = c / a;
        f.ty[q] = d / a;
    } else {
        f.tc[q] = 0.0;
        f.tp[q] = c;
        f.ty[q] = d;
    }
}

// With viscosity breaking MASK9 does not change once it is set, and with it
// the matrices stay: den and c' of every row depend on Depth, MASK9 and MASK
// alone.  k_thomas_fac walks the lines once per change (m9_dirty) and keeps c'
// and RN(1/den), and for periodic lines the second solution (tq); the solves
// (k_thomas_solve) then divide by den through its reciprocal
// (div_rcp: the same rounding), which leaves one sum, one product and two
// fused operations of each row on a line's critical path, and k_thomas_rows
// prepares d/a alone.  A den outside div_rcp's range keeps 0 for its
// reciprocal and is divided by.
// The planes are those that only the mixed mode's dispersion terms use.
template <typename T, int DIR> __device__ __forceinline__ double *tf_c(const Fields<T> &f) { return (double *)(DIR == 0 ? f.A : f.C); }
template <typename T, int DIR> __device__ __forceinline__ double *tf_y(const Fields<T> &f) { return (double *)(DIR == 0 ? f.B : f.E); }

// a, c, 1 + c_end or 1 + a_beg (the scale of a periodic line's end rows, else
// 1) and tmp2 of row k
template <typename T, int DIR, bool PER>
__device__ __forceinline__ void thomas_row(const Grid &g, const Fields<T> &f, const LinePart &lp, int i, int j, double &a,
                                           double &c, double &sc) {
    const int k = DIR == 0 ? i - g.ib : j - g.jb;
    double d;
    tri_coef<T, DIR>(g, f, i, j, a, c, d);
    sc = 1.0;
    if (PER && (k == 0 || k == lp.L - 1)) {
        double a2, c2;
        const bool first = k == 0;
        tri_coef<T, DIR>(g, f, DIR == 0 ? (first ? g.ie : g.ib) : i, DIR == 0 ? j : (first ? g.je : g.jb), a2, c2, d);
        sc = 1 + (first ? c2 : a2);
        if (first) c = c / sc;
        else a = a / sc;
    }
}

template <typename T, int DIR, bool PER>
__device__ __forceinline__ void thomas_ends(const Grid &g, const Fields<T> &f, const LinePart &lp, int l, double &a_beg, double &c_end) {
    double a, c, d;
    int i, j;
    line_cell<DIR>(g, l, 0, i, j);
    tri_coef<T, DIR>(g, f, i, j, a, c, d);
    a_beg = a;
    line_cell<DIR>(g, l, lp.L - 1, i, j);
    tri_coef<T, DIR>(g, f, i, j, a, c, d);
    c_end = c;
}
template <typename T, int DIR, bool PER>
__device__ void thomas_fac_body(const Grid &g, const Fields<T> &f, const LinePart &lp, int l) {
    if (l >= lp.nlines) return;
    double *FC = tf_c<T, DIR>(f), *FY = tf_y<T, DIR>(f);
    double cp = 0.0, ep = 0.0, e_first = 0.0, e_last = 0.0;
    if (PER) {
        // e = [1/(1+c_end), 0, ..., 0, -1/(1+a_beg)] (tridiagnal.F:207-215)
        double a_beg, c_end;
        thomas_ends<T, DIR, PER>(g, f, lp, l, a_beg, c_end);
        e_first = 1.0 / (1.0 + c_end);
        e_last = -1.0 / (1.0 + a_beg);
    }
    for (int k = 0; k < lp.L; k++) {
        int i, j;
        line_cell<DIR>(g, l, k, i, j);
        double a, c, sc;
        thomas_row<T, DIR, PER>(g, f, lp, i, j, a, c, sc);
        double y = 0.0;
        if (k > 0 && a != 0.0) {
            const double den = 1.0 / a - cp;
            cp = (c / a) / den;
            if (div_rcp_ok(den)) y = 1.0 / den;
            // e/a: 0/a is a zero with the sign of a; the last row's a is scaled
            if (PER) ep = ((k == lp.L - 1 ? e_last / a : fcopysign(0.0, a)) - ep) / den;
        } else {
            cp = c;
            if (PER) ep = k == lp.L - 1 ? e_last : (k == 0 ? e_first : 0.0);
        }
        FC[IDX(i, j)] = cp;
        FY[IDX(i, j)] = y;
        if (PER) f.tq[IDX(i, j)] = ep;
    }
    if (PER)
        for (int k = lp.L - 2; k >= 0; k--) {
            int i, j;
            line_cell<DIR>(g, l, k, i, j);
            ep = f.tq[IDX(i, j)] - FC[IDX(i, j)] * ep;
            f.tq[IDX(i, j)] = ep;
        }
}
// both directions in one launch: blocks [0, nbx) factor x, the rest y
template <typename T, bool PERY>
__global__ void __launch_bounds__(32) k_thomas_fac(Grid g, Fields<T> f, LinePart px, LinePart py, int nbx) {
    if (!*f.m9_dirty) return;
    if ((int)blockIdx.x < nbx) thomas_fac_body<T, 0, false>(g, f, px, blockIdx.x * 32 + threadIdx.x);
    else thomas_fac_body<T, 1, PERY>(g, f, py, (blockIdx.x - nbx) * 32 + threadIdx.x);
}

// the planes of 1/a and of d/a: each direction its own, so that both can be
// solved at once, and neither in its right-hand side's place, so that a solve
// can be repeated.  (Vyy: read by k_disp_b alone, which has run by then, and
// written anew before it runs again.)
template <typename T, int DIR> __device__ __forceinline__ double *tf_ra(const Fields<T> &f) { return DIR == 0 ? f.tc : f.tp; }
template <typename T, int DIR> __device__ __forceinline__ double *tf_d(const Fields<T> &f) {
    return DIR == 0 ? f.ty : reinterpret_cast<double *>(f.Vyy);
}
// d/a (or d) and 1/a (or 0) of every row, as k_thomas_rows
template <typename T, int DIR, bool PER>
__global__ void __launch_bounds__(256) k_thomas_rhs(Grid g, Fields<T> f, LinePart lp, int clear_dirty) {
    if (clear_dirty && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && threadIdx.y == 0) *f.m9_dirty = 0;
    const int i = g.ib + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = g.jb + blockIdx.y * blockDim.y + threadIdx.y;
    if (i > g.ie || j > g.je) return;
    const size_t q = IDX(i, j);
    const int k = DIR == 0 ? i - g.ib : j - g.jb;
    // tri_coef's a and d; tmp2 > 0 here (the launcher's condition)
    const double mdf = g.min_depth_frc, g1 = g.gamma1;
    const double dep = tmax((double)ro(f.Depth + q), mdf);
    const double depl = tmax((double)ro(f.Depth + (DIR == 0 ? IDX(i - 1, j) : IDX(i, j - 1))), mdf);
    const double m9 = ro(f.MASK9 + q) ? 1.0 : 0.0;
    const double tmp4 = DIR == 0 ? f.rhs_x[q] : f.rhs_y[q];
    const double k1 = g.tK1[DIR], k2 = g.tK2[DIR], k3 = g.tK3[DIR], k4 = g.tK4[DIR];
    const double gm = g1 * m9;
    const double tmp1 = gm * (k1 * dep * dep + k2 * depl * dep);
    const double tmp2 = 1.0 + gm * (k3 * dep * dep - k4 * dep * dep);
    const double r2 = __drcp_rn(tmp2);
    const bool ok = div_rcp_ok(tmp2);
    double a = ok ? div_rcp(tmp1, tmp2, r2) : tmp1 / tmp2, d = ok ? div_rcp(tmp4, tmp2, r2) : tmp4 / tmp2;
    if (PER && (k == 0 || k == lp.L - 1)) {
        double a2, c2, sc;
        thomas_row<T, DIR, PER>(g, f, lp, i, j, a2, c2, sc);
        if (k > 0) a = a / sc;
        d = d / sc;
    }
    double ra = 0.0;
    if (k > 0 && a != 0.0) {
        ra = __drcp_rn(a);
        d = div_rcp_ok(a) ? div_rcp(d, a, ra) : d / a;
    }
    tf_ra<T, DIR>(f)[q] = ra;
    tf_d<T, DIR>(f)[q] = d;
}

template <typename T, int DIR, bool PER>
__global__ void __launch_bounds__(32) k_thomas_lines(Grid g, Fields<T> f, LinePart lp) {
    constexpr int U = 8;  // rows per block of loads
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= lp.nlines) return;
    const int L = lp.L;
    const size_t base = DIR == 0 ? IDX(g.ib, g.jb + l) : IDX(g.ib + l, g.jb);
    const size_t step = DIR == 0 ? 1 : (size_t)g.pitch;
    double a_beg = 0.0, c_end = 0.0, e_first = 0.0, e_last = 0.0, ea_last = 0.0;
    if (PER) {
        double a, c, d;
        int i, j;
        line_cell<DIR>(g, l, 0, i, j);
        tri_coef<T, DIR>(g, f, i, j, a, c, d);
        a_beg = a;
        line_cell<DIR>(g, l, L - 1, i, j);
        tri_coef<T, DIR>(g, f, i, j, a, c, d);
        c_end = c;
        // e = [1/(1+c_end), 0, ..., 0, -1/(1+a_beg)] (tridiagnal.F:207-215);
        // the last row eliminates e/a with its scaled a
        e_first = 1.0 / (1.0 + c_end);
        e_last = -1.0 / (1.0 + a_beg);
        ea_last = e_last / (a / (1 + a_beg));
    }
    double cra[U], cca[U], cda[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        const size_t q = base + (size_t)u * step;
        cra[u] = u < L ? f.tc[q] : 0.0;
        cca[u] = u < L ? f.tp[q] : 0.0;
        cda[u] = u < L ? f.ty[q] : 0.0;
    }
    double cp = 0.0, dp = 0.0, ep = 0.0;
    for (int k0 = 0; k0 < L; k0 += U) {
        double nra[U], nca[U], nda[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int kk = k0 + U + u;
            const size_t q = base + (size_t)kk * step;
            nra[u] = kk < L ? f.tc[q] : 0.0;
            nca[u] = kk < L ? f.tp[q] : 0.0;
            nda[u] = kk < L ? f.ty[q] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int k = k0 + u;
            if (k < L) {
                double c, d, e = 0.0;
                if (cra[u] != 0.0) {
                    const double den = cra[u] - cp;
                    c = cca[u] / den;
                    d = (cda[u] - dp) / den;
                    // e/a: 0/a is a zero with the sign of a (that of 1/a)
                    if (PER) e = ((k == L - 1 ? ea_last : fcopysign(0.0, cra[u])) - ep) / den;
                } else {
                    c = cca[u];
                    d = cda[u];
                    if (PER) e = k == L - 1 ? e_last : (k == 0 ? e_first : 0.0);
                }
                cp = c;
                dp = d;
                ep = e;
                const size_t q = base + (size_t)k * step;
                f.tp[q] = c;
                f.ty[q] = d;
                if (PER) f.tq[q] = e;
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            cra[u] = nra[u];
            cca[u] = nca[u];
            cda[u] = nda[u];
        }
    }
    // back substitution, blocks of U rows from the end; the first solution
    // into ty, the second into tq (periodic), else straight into U / V
    T *out = DIR == 0 ? f.U : f.V;
    double z1 = 0.0, z2 = 0.0;
    const int nblk = (L + U - 1) / U;
    double ccp[U], cdp[U], cep[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int k = L - 1 - u;
        const size_t q = base + (size_t)(k >= 0 ? k : 0) * step;
        ccp[u] = k >= 0 ? f.tp[q] : 0.0;
        cdp[u] = k >= 0 ? f.ty[q] : 0.0;
        cep[u] = (PER && k >= 0) ? f.tq[q] : 0.0;
    }
    for (int b = 0; b < nblk; b++) {
        double ncp[U], ndp[U], nep[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int k = L - 1 - (b + 1) * U - u;
            const size_t q = base + (size_t)(k >= 0 ? k : 0) * step;
            ncp[u] = k >= 0 ? f.tp[q] : 0.0;
            ndp[u] = k >= 0 ? f.ty[q] : 0.0;
            nep[u] = (PER && k >= 0) ? f.tq[q] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int k = L - 1 - b * U - u;
            if (k >= 0) {
                if (k == L - 1) {
                    z1 = cdp[u];
                    if (PER) z2 = cep[u];
                } else {
                    z1 = cdp[u] - ccp[u] * z1;
                    if (PER) z2 = cep[u] - ccp[u] * z2;
                }
                const size_t q = base + (size_t)k * step;
                if (PER) {
                    f.ty[q] = z1;
                    f.tq[q] = z2;
                } else {
                    out[q] = (T)z1;
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            ccp[u] = ncp[u];
            cdp[u] = ndp[u];
            cep[u] = nep[u];
        }
    }
    if (PER) {
        const size_t q0 = base, q1 = base + (size_t)(L - 1) * step;
        const double beta = (c_end * f.ty[q0] - a_beg * f.ty[q1]) / (1.0 - (c_end * f.tq[q0] - a_beg * f.tq[q1]));
        for (int k = 0; k < L; k++) {
            const size_t q = base + (size_t)k * step;
            out[q] = (T)(f.ty[q] + beta * f.tq[q]);
        }
    }
}

// The solves with the kept factors: one warp walks 32 lines.  A line's chain
// is d'(k) = (d/a - d'(k-1)) / den: rows are worked in blocks of eight without
// a branch, with the next block's loads in flight, and a block that holds a
// row that is not eliminated, or a numerator outside div_rcp's range, is
// worked again row by row.  For periodic lines the second solution is kept
// (tq) and every warp of the block adds it at the end.
// Measured with the launches beside it (us, before -> after): 701 x 937 x 650
// -> 326, y 1326 -> 360; 250 x 500, periodic y, x 232 -> 120, y 1262 -> 219.
// What bounds it is the chain: four dependent FP64 operations a row forward
// and two back.
constexpr int THS_WARPS = 8;  // warps of a block of periodic lines
template <typename T, int DIR, bool PER>
__global__ void __launch_bounds__(PER ? 32 * THS_WARPS : 32) k_thomas_solve(Grid g, Fields<T> f, LinePart lp) {
    constexpr int U = 8;
    const int l = blockIdx.x * 32 + threadIdx.x, L = lp.L;
    const bool on = l < lp.nlines;
    const int base = (int)(DIR == 0 ? IDX(g.ib, g.jb + (on ? l : 0)) : IDX(g.ib + (on ? l : 0), g.jb));
    const int step = DIR == 0 ? 1 : g.pitch;
    T *const out = (DIR == 0 ? f.U : f.V) + base;
    double *const dp_ = tf_d<T, DIR>(f) + base;
    if (on && threadIdx.y == 0) {
        const double *const ra_ = tf_ra<T, DIR>(f) + base, *const fc_ = tf_c<T, DIR>(f) + base, *const fy_ = tf_y<T, DIR>(f) + base;
        double cp = 0.0, dp = 0.0;
        // one row as k_thomas_lines
        auto row = [&](double ra, double da, double fc, double fy) {
            double d = da;
            if (ra != 0.0) {
                const double den = ra - cp;
                d = fy != 0.0 ? div_rcp(da - dp, den, fy) : (da - dp) / den;
            }
            cp = fc;
            dp = d;
        };
        const int nb = L / U;
        double ra[U], da[U], fc[U], fy[U];
        auto load = [&](double *a, double *b, double *c, double *d, int k0) {
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int q = (k0 + u) * step;
                a[u] = ra_[q];
                b[u] = dp_[q];
                c[u] = fc_[q];
                d[u] = fy_[q];
            }
        };
        if (nb > 0) load(ra, da, fc, fy, 0);
        for (int b = 0; b < nb; b++) {
            double nra[U], nda[U], nfc[U], nfy[U];
            load(nra, nda, nfc, nfy, b + 1 < nb ? (b + 1) * U : b * U);
            double dv[U], c0 = cp, d0 = dp;
            unsigned bad = 0;
#pragma unroll
            for (int u = 0; u < U; u++) {
                const double den = ra[u] - c0, t = da[u] - d0, y = fy[u];
                const double q = __dmul_rn(t, y);
                dv[u] = d0 = __fma_rn(__fma_rn(-q, den, t), y, q);
                c0 = fc[u];
                // exponents of t and y (both high words); a zero t divides
                // right when y < 0
                const int th = __double2hiint(t), yh = __double2hiint(y);
                const unsigned te = (unsigned)th & 0x7fffffffu;
                const bool zero = (te | (unsigned)__double2loint(t)) == 0 && yh < 0;
                if ((yh << 1) == 0 || (te - ((1023u - 500u) << 20) >= (1000u << 20) && !zero)) bad = 1;
            }
            if (bad) {
#pragma unroll
                for (int u = 0; u < U; u++) {
                    row(ra[u], da[u], fc[u], fy[u]);
                    dv[u] = dp;
                }
            } else {
                cp = c0;
                dp = d0;
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                dp_[(b * U + u) * step] = dv[u];
                ra[u] = nra[u];
                da[u] = nda[u];
                fc[u] = nfc[u];
                fy[u] = nfy[u];
            }
        }
        for (int k = nb * U; k < L; k++) {
            const int q = k * step;
            row(ra_[q], dp_[q], fc_[q], fy_[q]);
            dp_[q] = dp;
        }
        // back substitution: the first solution into d's place (periodic), else
        // straight into U / V
        double z = dp;
        auto put = [&](int k, double v) {
            if (PER) dp_[k * step] = v;
            else out[k * step] = (T)v;
        };
        put(L - 1, z);
        int k = L - 2;
        double d1[U], c1[U];
        auto back = [&](double *d, double *c, int k0) {
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int q = max(k0 - u, 0) * step;
                d[u] = dp_[q];
                c[u] = fc_[q];
            }
        };
        back(d1, c1, k);
        for (; k >= U - 1; k -= U) {
            double d2[U], c2[U];
            back(d2, c2, k - U);
#pragma unroll
            for (int u = 0; u < U; u++) {
                z = d1[u] - c1[u] * z;
                put(k - u, z);
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                d1[u] = d2[u];
                c1[u] = c2[u];
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++)
            if (k - u >= 0) {
                z = d1[u] - c1[u] * z;
                put(k - u, z);
            }
    }
    if (PER) {
        __shared__ double beta_[32];
        if (on && threadIdx.y == 0) {
            double a_beg, c_end;
            thomas_ends<T, DIR, PER>(g, f, lp, l, a_beg, c_end);
            const double *z2 = f.tq + base;
            const int e = (L - 1) * step;
            beta_[threadIdx.x] = (c_end * dp_[0] - a_beg * dp_[e]) / (1.0 - (c_end * z2[0] - a_beg * z2[e]));
        }
        __syncthreads();
        if (on) {
            const double beta = beta_[threadIdx.x];
            const double *z2 = f.tq + base;
#pragma unroll 4
            for (int k = threadIdx.y; k < L; k += THS_WARPS) out[k * step] = (T)(__ldcg(dp_ + k * step) + beta * ro(z2 + k * step));
        }
    }
}

// Mixed path: the tridiagonal matrices depend on Depth and MASK9 only, so
// their partitioned factorisation is computed (in double) when MASK9 has
// changed or one of them was set - never again in a run with viscosity
// breaking once that has set MASK9 = 1 on the ring - and stored rounded to
// float.  Each stage then solves in float and
// refines once: x0 = S(d), r = d - T x0 with a compensated (float-pair)
// residual, x = x0 + S(r).  S is the partitioned substitution: per chunk of
// m rows a forward/backward sweep, a reduced system of two rows per chunk,
// and the interior recovery x_k = y_k - p_k x_s - q_k x_e.  For periodic y,
// S applies TRIDy_periodic's end-row scaling and Sherman-Morrison
// combination, whose result solves the cyclic system
// x0 + c0 x1 + a0 x(L-1) = d0, a(L-1) x(L-2) + x(L-1) + c(L-1) x0 = d(L-1)
// (tridiagnal.F:59-325); the residual uses that cyclic operator.
struct FacLine {
    float *lo, *di, *up, *cs, *ae, *x2, *tail;  // reduced rows; tail: c_end, a_beg, den_beta
};
__device__ __forceinline__ FacLine fac_line(float *base, const LinePart &lp, int l) {
    const int n = 2 * lp.P;
    float *b = base + (size_t)l * (size_t)(4 * n + 2 * lp.P + 3);
    FacLine f;
    f.lo = b;
    f.di = b + n;
    f.up = b + 2 * n;
    f.cs = b + 3 * n;
    f.ae = b + 3 * n + lp.P;
    f.x2 = b + 3 * n + 2 * lp.P;
    f.tail = b + 4 * n + 2 * lp.P;
    return f;
}

// normalised a, c and 1/tmp2 of one row, in double (no right-hand side)
template <typename T, int DIR>
__device__ __forceinline__ void tri_ac(const Grid &g, const Fields<T> &f, int i, int j, double &a, double &c,
                                       double &it) {
    const double mdf = g.min_depth_frc;
    const size_t id = IDX(i, j);
    const double dep = tmax((double)f.Depth[id], mdf);
    const double depl = tmax((double)f.Depth[DIR == 0 ? IDX(i - 1, j) : IDX(i, j - 1)], mdf);
    const double depr = tmax((double)f.Depth[DIR == 0 ? IDX(i + 1, j) : IDX(i, j + 1)], mdf);
    const double gm = g.gamma1 * (double)f.MASK9[id];
    const double tmp1 = gm * dep * (g.cA[DIR] * dep + g.cB[DIR] * depl);
    const double tmp2 = 1.0 + gm * g.cC[DIR] * dep * dep;
    const double tmp3 = gm * dep * (g.cA[DIR] * dep + g.cB[DIR] * depr);
    it = 1.0 / tmp2;
    a = tmp1 * it;
    c = tmp3 * it;
}

// a, c of row k with the periodic end-row scaling (tridiagnal.F:168-173)
template <typename T, int DIR, bool PER>
__device__ __forceinline__ void tri_ac_row(const Grid &g, const Fields<T> &f, const LinePart &lp, int l, int k,
                                           double &a, double &c, double &it) {
    int i, j;
    line_cell<DIR>(g, l, k, i, j);
    tri_ac<T, DIR>(g, f, i, j, a, c, it);
    if (PER && (k == 0 || k == lp.L - 1)) {
        double a2, c2, it2;
        int i2, j2;
        line_cell<DIR>(g, l, k == 0 ? lp.L - 1 : 0, i2, j2);
        tri_ac<T, DIR>(g, f, i2, j2, a2, c2, it2);
        if (k == 0) c = c / (1 + c2);   // c_end
        else a = a / (1 + a2);           // a_beg
    }
}

// where row k of line l keeps its factors: its cell, except that the x lines
// of LSF_M-row chunks keep the rows of equal offset in their chunks side by
// side, so that neighbouring threads, which own neighbouring chunks, load
// neighbouring words; the last chunk's rows past LSF_M keep their place
template <int DIR> __device__ __forceinline__ size_t fac_at(const Grid &g, const LinePart &lp, int l, int k) {
    if (DIR == 1) return IDX(g.ib + l, g.jb + k);
    const size_t row = (size_t)(g.jb + l) * g.pitch;
    if (lp.m != LSF_M) return row + g.ib + k;
    return row + (k < LSF_M * lp.P ? (k % LSF_M) * lp.P + k / LSF_M : k);
}

__device__ __forceinline__ void split2(double v, float &hi, float &lo) {
    hi = (float)v;
    lo = (float)(v - (double)hi);
}

template <typename T, int DIR, bool PER>
__device__ __forceinline__ void fac_a_body(const Grid &g, const Fields<T> &f, const LinePart &lp, int t) {
    if (t >= lp.nlines * lp.P) return;
    int l, ch;
    chunk_of<DIR>(lp, t, l, ch);
    const int s = ch * lp.m;
    const int e = (ch == lp.P - 1) ? lp.L - 1 : s + lp.m - 1;
    float *it_ = f.fac_it[DIR], *A_ = f.fac_A[DIR], *lr_ = f.fac_lr[DIR], *cp_ = f.fac_cp[DIR];
    float *p_ = f.fac_p[DIR], *q_ = f.fac_q[DIR];
    // the unscaled normalised coefficients of every row, for the residual
    for (int k = s; k <= e; k++) {
        double a, c, it;
        int i, j;
        line_cell<DIR>(g, l, k, i, j);
        tri_ac<T, DIR>(g, f, i, j, a, c, it);
        if (!PER && k == 0) a = 0.0;
        if (!PER && k == lp.L - 1) c = 0.0;
        const size_t q = fac_at<DIR>(g, lp, l, k);
        split2(a, f.fac_ah[DIR][q], f.fac_al[DIR][q]);
        split2(c, f.fac_ch[DIR][q], f.fac_cl[DIR][q]);
        it_[q] = (float)it;
    }
    double as, cs, its, ae, ce, ite;
    tri_ac_row<T, DIR, PER>(g, f, lp, l, s, as, cs, its);
    tri_ac_row<T, DIR, PER>(g, f, lp, l, e, ae, ce, ite);
    // a chunk's first and last row: constants with which the sweeps pass them by
    for (int k = s; k <= e; k += max(1, e - s)) {
        const size_t q = fac_at<DIR>(g, lp, l, k);
        A_[q] = 1.0f;
        lr_[q] = cp_[q] = p_[q] = q_[q] = 0.0f;
    }
    if (s == 0) as = 0.0;
    if (e == lp.L - 1) ce = 0.0;
    double lo_s, di_s, up_s, lo_e, di_e, up_e;
    if (e - s >= 2) {
        double cp = 0.0, pp = 0.0, qp = 0.0;
        double *pbuf = f.sw_p[DIR], *qbuf = f.sw_q[DIR], *cbuf = f.sw_c[DIR];  // sweep scratch of this direction
        for (int k = s + 1; k <= e - 1; k++) {
            double a, c, it;
            tri_ac_row<T, DIR, PER>(g, f, lp, l, k, a, c, it);
            const double lower = (k > s + 1) ? a : 0.0;
            const double r = 1.0 / (1.0 - lower * cp);
            const double upper = (k < e - 1) ? c : 0.0;
            cp = upper * r;
            pp = ((k == s + 1 ? a : 0.0) - lower * pp) * r;
            qp = ((k == e - 1 ? c : 0.0) - lower * qp) * r;
            const size_t q = fac_at<DIR>(g, lp, l, k);
            A_[q] = (float)r;
            lr_[q] = (float)(lower * r);
            cp_[q] = (float)cp;
            cbuf[q] = cp;
            pbuf[q] = pp;
            qbuf[q] = qp;
        }
        double pn = 0.0, qn = 0.0, p1 = 0.0, q1 = 0.0, pl = 0.0, ql = 0.0;
        for (int k = e - 1; k >= s + 1; k--) {
            const size_t q = fac_at<DIR>(g, lp, l, k);
            const double cpk = cbuf[q];
            const double pk = pbuf[q] - cpk * pn, qk = qbuf[q] - cpk * qn;
            p_[q] = (float)pk;
            q_[q] = (float)qk;
            pn = pk;
            qn = qk;
            if (k == e - 1) {
                pl = pk;
                ql = qk;
            }
            if (k == s + 1) {
                p1 = pk;
                q1 = qk;
            }
        }
        lo_s = as;
        di_s = 1.0 - cs * p1;
        up_s = -cs * q1;
        lo_e = -ae * pl;
        di_e = 1.0 - ae * ql;
        up_e = ce;
    } else {
        lo_s = as;
        di_s = 1.0;
        up_s = cs;
        lo_e = ae;
        di_e = 1.0;
        up_e = ce;
    }
    // reduced rows to the double scratch; k_fac_b factors them
    double *red = f.red + lp.red0 + ((size_t)l * 2 * lp.P + 2 * ch) * 6;
    red[0] = lo_s;
    red[1] = di_s;
    red[2] = up_s;
    red[6] = lo_e;
    red[7] = di_e;
    red[8] = up_e;
    FacLine fl = fac_line(f.fac_red[DIR], lp, l);
    fl.cs[ch] = (e - s >= 2) ? (float)cs : 0.0f;
    fl.ae[ch] = (e - s >= 2) ? (float)ae : 0.0f;
}

template <typename T, int DIR, bool PER>
__global__ void __launch_bounds__(128) k_fac_a(Grid g, Fields<T> f, LinePart lp) {
    if (!*f.m9_dirty) return;
    fac_a_body<T, DIR, PER>(g, f, lp, blockIdx.x * blockDim.x + threadIdx.x);
}

template <typename T, int DIR, bool PER>
__device__ __forceinline__ void fac_b_body(const Grid &g, const Fields<T> &f, const LinePart &lp, int l) {
    if (l >= lp.nlines) return;
    const int n = 2 * lp.P;
    double *red = f.red + lp.red0 + (size_t)l * n * 6;
    FacLine fl = fac_line(f.fac_red[DIR], lp, l);
    double cpr = 0.0;
    for (int k = 0; k < n; k++) {
        const double lo = (k > 0) ? red[k * 6 + 0] : 0.0;
        const double up = (k < n - 1) ? red[k * 6 + 2] : 0.0;
        const double id = 1.0 / (red[k * 6 + 1] - lo * cpr);
        cpr = up * id;
        fl.lo[k] = (float)lo;       // the reduced rows, solved per stage by
        fl.di[k] = (float)red[k * 6 + 1];  // parallel cyclic reduction
        fl.up[k] = (float)up;
        red[k * 6 + 3] = lo;   // double factors for the periodic solve below
        red[k * 6 + 4] = id;
        red[k * 6 + 5] = cpr;
    }
    if (PER) {
        // the second periodic solution (right-hand side e of TRIDy_periodic,
        // tridiagnal.F:207-215) and the constant denominator of beta
        double a, c, it;
        int i, j;
        line_cell<DIR>(g, l, 0, i, j);
        tri_ac<T, DIR>(g, f, i, j, a, c, it);
        const double a_beg = a;
        line_cell<DIR>(g, l, lp.L - 1, i, j);
        tri_ac<T, DIR>(g, f, i, j, a, c, it);
        const double c_end = c;
        double z = 0.0;
        for (int k = 0; k < n; k++) {
            const double rhs = k == 0 ? 1.0 / (1.0 + c_end) : (k == n - 1 ? -1.0 / (1.0 + a_beg) : 0.0);
            z = (rhs - red[k * 6 + 3] * z) * red[k * 6 + 4];
            red[k * 6 + 4] = z;
        }
        double x = 0.0, x0 = 0.0, xl = 0.0;
        for (int k = n - 1; k >= 0; k--) {
            x = red[k * 6 + 4] - red[k * 6 + 5] * x;
            fl.x2[k] = (float)x;
            if (k == n - 1) xl = x;
            if (k == 0) x0 = x;
        }
        fl.tail[0] = (float)c_end;
        fl.tail[1] = (float)a_beg;
        fl.tail[2] = (float)(1.0 - (c_end * x0 - a_beg * xl));
    }
}

// The multipliers of the parallel cyclic reduction of a line's reduced rows,
// constant like the factors (and computed with them: where MASK9 moves, at most
// stages; with k_linesolve such a step of 1024 x 1024 takes 2522 us, 2701 with
// the solves before it and no multipliers): per step a and b (n4 words each), then the last
// diagonal; the operations are pcr_solve's.  They lie in the planes that only
// the FP64 mode's dispersion terms use (eight consecutive planes from Uxx; at
// most 19/8 words per cell and direction), x lines first.
template <typename T, int DIR>
__device__ __forceinline__ float *pcr_line(const Fields<T> &f, const LinePart &lp, int l) {
    return (float *)f.Uxx + lp.pcr0 + (size_t)l * pcr_words(lp);
}
// one line by a block of 128 threads; sh: 6 x 2P words
template <typename T, int DIR>
__device__ void pcr_factor(const Fields<T> &f, const LinePart &lp, int l, float *sh) {
    const int n = 2 * lp.P, n4 = (n + 3) & ~3;
    const double *red = f.red + lp.red0 + (size_t)l * n * 6;
    float *out = pcr_line<T, DIR>(f, lp, l);
    float *lo = sh, *di = sh + n, *up = sh + 2 * n, *lo2 = sh + 3 * n, *di2 = sh + 4 * n, *up2 = sh + 5 * n;
    __syncthreads();  // the previous line's readers
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        lo[k] = (float)((k > 0) ? red[k * 6 + 0] : 0.0);
        di[k] = (float)red[k * 6 + 1];
        up[k] = (float)((k < n - 1) ? red[k * 6 + 2] : 0.0);
    }
    __syncthreads();
    for (int st = 1; st < n; st <<= 1) {
        for (int k = threadIdx.x; k < n; k += blockDim.x) {
            const int km = k - st, kp = k + st;
            float a = 0.0f, b = 0.0f, nlo = 0.0f, nup = 0.0f;
            float nd = di[k];
            if (km >= 0) {
                a = -lo[k] / di[km];
                nlo = a * lo[km];
                nd += a * up[km];
            }
            if (kp < n) {
                b = -up[k] / di[kp];
                nup = b * up[kp];
                nd += b * lo[kp];
            }
            lo2[k] = nlo;
            di2[k] = nd;
            up2[k] = nup;
            out[k] = a;
            out[n4 + k] = b;
        }
        out += 2 * n4;
        __syncthreads();
        float *t;
        t = lo; lo = lo2; lo2 = t;
        t = di; di = di2; di2 = t;
        t = up; up = up2; up2 = t;
    }
    for (int k = threadIdx.x; k < n; k += blockDim.x) out[k] = di[k];
}

// blocks [0, nb) factor the reduced rows, one line per thread; the others take
// the reduction's multipliers, one line per block at a time (both read words
// 0..2 of the reduced rows, and only the first write words 3..5)
template <typename T, int DIR, bool PER>
__global__ void __launch_bounds__(128) k_fac_b(Grid g, Fields<T> f, LinePart lp, int nb) {
    extern __shared__ float shp[];
    if (!*f.m9_dirty) return;
    if ((int)blockIdx.x < nb) {
        fac_b_body<T, DIR, PER>(g, f, lp, blockIdx.x * blockDim.x + threadIdx.x);
        return;
    }
    for (int l = blockIdx.x - nb; l < lp.nlines; l += gridDim.x - nb) pcr_factor<T, DIR>(f, lp, l, shp);
}

// both directions in one launch each: blocks [0, nbx) factor x, the rest y
template <typename T, bool PERY>
__global__ void __launch_bounds__(128) k_fac_a_xy(Grid g, Fields<T> f, LinePart px, LinePart py, int nbx) {
    if (!*f.m9_dirty) return;
    if ((int)blockIdx.x < nbx) fac_a_body<T, 0, false>(g, f, px, blockIdx.x * blockDim.x + threadIdx.x);
    else fac_a_body<T, 1, PERY>(g, f, py, (blockIdx.x - nbx) * blockDim.x + threadIdx.x);
}
template <typename T, bool PERY>
__global__ void __launch_bounds__(128) k_fac_b_xy(Grid g, Fields<T> f, LinePart px, LinePart py, int nbx, int nby) {
    extern __shared__ float shp[];
    if (!*f.m9_dirty) return;
    const int b = blockIdx.x - nbx - nby;
    if ((int)blockIdx.x < nbx) {
        fac_b_body<T, 0, false>(g, f, px, blockIdx.x * blockDim.x + threadIdx.x);
    } else if (b < 0) {
        fac_b_body<T, 1, PERY>(g, f, py, (blockIdx.x - nbx) * blockDim.x + threadIdx.x);
    } else {
        const int nx = lsf_line(px) ? px.nlines : 0, ny = lsf_line(py) ? py.nlines : 0;
        for (int l = b; l < nx + ny; l += gridDim.x - nbx - nby) {
            if (l < nx) pcr_factor<T, 0>(f, px, l, shp);
            else pcr_factor<T, 1>(f, py, l - nx, shp);
        }
    }
}

static __global__ void k_fac_clear(int *dirty) { *dirty = 0; }

// compensated r = d - (a x(k-1) + x(k) + c x(k+1)) with a = ah + al, c = ch + cl
// Every operation is written as rounded (no contraction left to the
// compiler), so that all callers get the same bits.
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e) {
    s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}
__device__ __forceinline__ void two_prod(float a, float b, float &p, float &e) {
    p = __fmul_rn(a, b);
    e = __fmaf_rn(a, b, -p);
}
__device__ __forceinline__ float residual(float d, float x, float xm, float xp, float ah, float al, float ch,
                                          float cl) {
    float t, e1, u, e2, v, e3, t2, e4, t3, e5;
    two_sum(d, -x, t, e1);
    two_prod(ah, xm, u, e2);
    two_prod(ch, xp, v, e3);
    two_sum(t, -u, t2, e4);
    two_sum(t2, -v, t3, e5);
    const float lo = __fsub_rn(__fsub_rn(__fadd_rn(__fadd_rn(e1, e4), e5), e2), e3);
    return __fadd_rn(t3, __fmaf_rn(-cl, xp, __fmaf_rn(-al, xm, lo)));
}

// Parallel cyclic reduction of n reduced rows lo x(k-1) + di x(k) +
// up x(k+1) = r in shared memory by the whole block: log2(n) steps, each row
// eliminating its neighbours at distance s; the solution replaces r.
// Buffers: lo, di, up, r and their doubles lo2, di2, up2, r2 (n floats each).
__device__ __forceinline__ void pcr_solve(float *lo, float *di, float *up, float *r, float *lo2, float *di2,
                                          float *up2, float *r2, int n) {
    for (int st = 1; st < n; st <<= 1) {
        for (int k = threadIdx.x; k < n; k += blockDim.x) {
            const int km = k - st, kp = k + st;
            float a = 0.0f, b = 0.0f, nlo = 0.0f, nup = 0.0f;
            float nd = di[k], nr = r[k];
            if (km >= 0) {
                a = -lo[k] / di[km];
                nlo = a * lo[km];
                nd += a * up[km];
                nr += a * r[km];
            }
            if (kp < n) {
                b = -up[k] / di[kp];
                nup = b * up[kp];
                nd += b * lo[kp];
                nr += b * r[kp];
            }
            lo2[k] = nlo;
            di2[k] = nd;
            up2[k] = nup;
            r2[k] = nr;
        }
        __syncthreads();
        float *t;
        t = lo; lo = lo2; lo2 = t;
        t = di; di = di2; di2 = t;
        t = up; up = up2; up2 = t;
        t = r; r = r2; r2 = t;
    }
    // after the last swap the current buffers may be the doubles: copy the
    // solution into both
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const float x = r[k] / di[k];
        r[k] = x;
        r2[k] = x;
    }
    __syncthreads();
}

// y lines (and the periodic direction): per-chunk kernels, coalesced across
// neighbouring lines.  PASS 0 solves d = rhs/tmp2, PASS 1 the residual.
// per-stage reduced right-hand sides: pass 0 at the start of the scratch,
// pass 1 right after it
template <int PASS> __device__ __forceinline__ float *red_rhs(double *red, const LinePart &lp) {
    return (float *)red + (PASS == 0 ? 0 : (size_t)lp.nlines * 2 * lp.P);
}

template <typename T, int DIR, bool PER, int PASS>
__global__ void __launch_bounds__(128) k_sol_a(Grid g, Fields<T> f, LinePart lp) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= lp.nlines * lp.P) return;
    int l, ch;
    chunk_of<DIR>(lp, t, l, ch);
    const int s = ch * lp.m;
    const int e = (ch == lp.P - 1) ? lp.L - 1 : s + lp.m - 1;
    const T *rhs = DIR == 0 ? f.rhs_x : f.rhs_y;
    const float *it_ = f.fac_it[DIR], *A_ = f.fac_A[DIR], *lr_ = f.fac_lr[DIR], *cp_ = f.fac_cp[DIR];
    float *ys = (float *)f.ty;   // y of this pass
    const float *rr = (const float *)f.tq;  // residual (PASS 1)
    FacLine fl = fac_line(f.fac_red[DIR], lp, l);
    float sc0 = 1.0f, sc1 = 1.0f;
    if (PER) {
        sc0 = 1.0f / (1.0f + fl.tail[0]);  // row 0: d / (1 + c_end)
        sc1 = 1.0f / (1.0f + fl.tail[1]);  // row L-1: d / (1 + a_beg)
    }
    auto dval = [&](int k, size_t q) {
        float d = PASS == 0 ? (float)rhs[q] * it_[q] : rr[q];
        if (PER && k == 0) d *= sc0;
        if (PER && k == lp.L - 1) d *= sc1;
        return d;
    };
    int i, j;
    line_cell<DIR>(g, l, s, i, j);
    const float ds = dval(s, IDX(i, j));
    line_cell<DIR>(g, l, e, i, j);
    const float de = dval(e, IDX(i, j));
    float rs = ds, re = de;
    if (e - s >= 2) {
        float yp = 0.0f;
        for (int k = s + 1; k <= e - 1; k++) {
            line_cell<DIR>(g, l, k, i, j);
            const size_t q = IDX(i, j);
            yp = dval(k, q) * A_[q] - lr_[q] * yp;
            ys[q] = yp;
        }
        float yn = 0.0f, y1 = 0.0f, yl = 0.0f;
        for (int k = e - 1; k >= s + 1; k--) {
            line_cell<DIR>(g, l, k, i, j);
            const size_t q = IDX(i, j);
            const float yk = ys[q] - cp_[q] * yn;
            ys[q] = yk;
            yn = yk;
            if (k == e - 1) yl = yk;
            if (k == s + 1) y1 = yk;
        }
        rs = ds - fl.cs[ch] * y1;
        re = de - fl.ae[ch] * yl;
    }
    float *red = red_rhs<PASS>(f.red, lp) + ((size_t)l * 2 * lp.P + 2 * ch);
    red[0] = rs;
    red[1] = re;
}

template <typename T, int DIR, bool PER, int PASS>
__global__ void __launch_bounds__(512) k_sol_b(Grid g, Fields<T> f, LinePart lp) {
    extern __shared__ float shr[];
    const int l = blockIdx.x;
    const int n = 2 * lp.P;
    float *red = red_rhs<PASS>(f.red, lp) + (size_t)l * n;
    FacLine fl = fac_line(f.fac_red[DIR], lp, l);
    float *lo = shr, *di = shr + n, *up = shr + 2 * n, *r = shr + 3 * n;
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        lo[k] = fl.lo[k];
        di[k] = fl.di[k];
        up[k] = fl.up[k];
        r[k] = red[k];
    }
    __syncthreads();
    pcr_solve(lo, di, up, r, shr + 4 * n, shr + 5 * n, shr + 6 * n, shr + 7 * n, n);
    float beta = 0.0f;
    if (PER) beta = (fl.tail[0] * r[0] - fl.tail[1] * r[n - 1]) / fl.tail[2];
    for (int k = threadIdx.x; k < n; k += blockDim.x) red[k] = PER ? r[k] + beta * fl.x2[k] : r[k];
}

// PASS 0: x0 -> tp scratch; PASS 1: out = x0 + correction
template <typename T, int DIR, int PASS>
__global__ void __launch_bounds__(128) k_sol_c(Grid g, Fields<T> f, LinePart lp) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= lp.nlines * lp.P) return;
    int l, ch;
    chunk_of<DIR>(lp, t, l, ch);
    const int s = ch * lp.m;
    const int e = (ch == lp.P - 1) ? lp.L - 1 : s + lp.m - 1;
    const float *red = red_rhs<PASS>(f.red, lp) + ((size_t)l * 2 * lp.P + 2 * ch);
    const float xs = red[0], xe = red[1];
    const float *p_ = f.fac_p[DIR], *q_ = f.fac_q[DIR];
    const float *ys = (const float *)f.ty;
    float *x0 = (float *)f.tp;
    T *out = DIR == 0 ? f.U : f.V;
    for (int k = s; k <= e; k++) {
        int i, j;
        line_cell<DIR>(g, l, k, i, j);
        const size_t q = IDX(i, j);
        const float x = (k == s) ? xs : (k == e) ? xe : ys[q] - p_[q] * xs - q_[q] * xe;
        if (PASS == 0) x0[q] = x;
        else out[q] = (T)(x0[q] + x);
    }
}

// compensated residual of the first solve on every interior cell
template <typename T, int DIR, bool PER>
__global__ void __launch_bounds__(256) k_resid(Grid g, Fields<T> f, LinePart lp) {
    const int i = g.ib + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = g.jb + blockIdx.y * blockDim.y + threadIdx.y;
    if (i > g.ie || j > g.je) return;
    const size_t q = IDX(i, j);
    const int k = DIR == 0 ? i - g.ib : j - g.jb;
    const size_t st = DIR == 0 ? 1 : (size_t)g.pitch;
    const float *x0 = (const float *)f.tp;
    const T *rhs = DIR == 0 ? f.rhs_x : f.rhs_y;
    const float d = (float)rhs[q] * f.fac_it[DIR][q];
    // neighbours along the line; the cyclic ends wrap in periodic y
    float xm = 0.0f, xp = 0.0f;
    if (k > 0) xm = x0[q - st];
    else if (PER) xm = x0[q + (size_t)(lp.L - 1) * st];
    if (k < lp.L - 1) xp = x0[q + st];
    else if (PER) xp = x0[q - (size_t)(lp.L - 1) * st];
    ((float *)f.tq)[q] = residual(d, x0[q], xm, xp, f.fac_ah[DIR][q], f.fac_al[DIR][q], f.fac_ch[DIR][q],
                                  f.fac_cl[DIR][q]);
}

// x lines, one block per line, everything unit-stride: load d, solve, form
// the compensated residual, solve again and write x0 + correction.  The
// arrays that a thread walks along its own chunk are stored with one pad
// float after every 16 (index k + k/16), so that the 32 chunks a warp walks
// at once fall into different shared-memory banks.
__host__ __device__ __forceinline__ int lsx_pad(int k) { return k + (k >> 4); }
__host__ __device__ __forceinline__ size_t lsx_smem_floats(int L, int P) {
    return (size_t)6 * (lsx_pad(L) + 1) + (size_t)L + 16 * (size_t)P;
}

template <typename T>
__global__ void __launch_bounds__(256) k_linesolve_x(Grid g, Fields<T> f, LinePart lp, int clear_dirty) {
    extern __shared__ float shf[];
    const int l = blockIdx.x;
    // the factorisation of this stage is complete: the MASK9 change flag
    // can be reset for UPDATE_MASK to set again
    if (clear_dirty && l == 0 && threadIdx.x == 0) *f.m9_dirty = 0;
    const int L = lp.L, P = lp.P, m = lp.m;
    const int LP = lsx_pad(L) + 1;
    float *d = shf;            // right-hand side, then residual (padded)
    float *y = shf + LP;       // sweep values (padded)
    float *A = shf + 2 * LP;   // sweep constants, staged with unit-stride loads (padded)
    float *LR = shf + 3 * LP;
    float *CP = shf + 4 * LP;
    float *dn = shf + 5 * LP;  // the normalised right-hand side, kept for the residual (padded)
    float *x0 = shf + 6 * LP;  // L  first solution (unpadded)
    float *rr = x0 + L;        // 2P reduced right-hand sides / solution
    float *pb = rr + 2 * P;    // 7 x 2P PCR buffers
    const int j = g.jb + l;
    const size_t row = (size_t)j * g.pitch + g.ib;
    const T *rhs = f.rhs_x + row;
    const float *IT = f.fac_it[0] + row, *Pp = f.fac_p[0] + row, *Qq = f.fac_q[0] + row;
    const float *AH = f.fac_ah[0] + row, *AL = f.fac_al[0] + row;
    const float *CH = f.fac_ch[0] + row, *CL = f.fac_cl[0] + row;
    FacLine fl = fac_line(f.fac_red[0], lp, l);
    const int ch = threadIdx.x;
    const int s = ch * m;
    const int e = (ch == P - 1) ? L - 1 : s + m - 1;
    const int n = 2 * P;
    for (int k = threadIdx.x; k < L; k += blockDim.x) {
        const int q = lsx_pad(k);
        const float dv = (float)rhs[k] * IT[k];
        d[q] = dv;
        dn[q] = dv;
        A[q] = f.fac_A[0][row + k];
        LR[q] = f.fac_lr[0][row + k];
        CP[q] = f.fac_cp[0][row + k];
    }
    __syncthreads();
    for (int pass = 0; pass < 2; pass++) {
        // chunk forward/backward sweeps
        if (ch < P) {
            float rs = d[lsx_pad(s)], re = d[lsx_pad(e)];
            if (e - s >= 2) {
                float yp = 0.0f;
                for (int k = s + 1; k <= e - 1; k++) {
                    const int q = lsx_pad(k);
                    yp = d[q] * A[q] - LR[q] * yp;
                    y[q] = yp;
                }
                float yn = 0.0f;
                for (int k = e - 1; k >= s + 1; k--) {
                    const int q = lsx_pad(k);
                    yn = y[q] - CP[q] * yn;
                    y[q] = yn;
                }
                rs = rs - fl.cs[ch] * y[lsx_pad(s + 1)];
                re = re - fl.ae[ch] * y[lsx_pad(e - 1)];
            }
            rr[2 * ch] = rs;
            rr[2 * ch + 1] = re;
        }
        for (int k = threadIdx.x; k < n; k += blockDim.x) {
            pb[k] = fl.lo[k];
            pb[n + k] = fl.di[k];
            pb[2 * n + k] = fl.up[k];
        }
        __syncthreads();
        pcr_solve(pb, pb + n, pb + 2 * n, rr, pb + 3 * n, pb + 4 * n, pb + 5 * n, pb + 6 * n, n);
        auto recon = [&](int k, float p_, float q_) {
            const int c = min(lp.lgm >= 0 ? k >> lp.lgm : k / m, P - 1);
            const int cs = c * m, ce = (c == P - 1) ? L - 1 : cs + m - 1;
            const float x = (k == cs) ? rr[2 * c] : (k == ce) ? rr[2 * c + 1] : y[lsx_pad(k)] - p_ * rr[2 * c] - q_ * rr[2 * c + 1];
            if (pass == 0) x0[k] = x;
            else f.U[row + k] = (T)(x0[k] + x);
        };
        for (int k = threadIdx.x; k < L; k += blockDim.x) recon(k, Pp[k], Qq[k]);
        __syncthreads();
        if (pass == 0) {
            auto resid = [&](int k, float ah, float al, float chv, float cl) {
                const float xm = k > 0 ? x0[k - 1] : 0.0f, xp = k < L - 1 ? x0[k + 1] : 0.0f;
                const int q = lsx_pad(k);
                d[q] = residual(dn[q], x0[k], xm, xp, ah, al, chv, cl);
            };
            for (int k = threadIdx.x; k < L; k += blockDim.x) resid(k, AH[k], AL[k], CH[k], CL[k]);
            __syncthreads();
        }
    }
}

// ---------------------------------------------------------------------------
// The mixed u/v recovery of one direction in one kernel, for lines of 32 to
// 4096 rows (chunks of LSF_M rows).  A thread owns one chunk of one line and
// keeps its rows in registers from the right-hand side to the result: sweeps,
// reduced system, reconstruction, compensated residual, and the same again on
// the residual.  HBM sees the right-hand side, the constant factors and the
// result once each: 56 B per cell.
//   x lines: a block takes a few whole lines.  Their factors lie chunk-
//   interleaved (fac_at), so the 32 chunks of a warp load neighbouring words;
//   the right-hand side and the result cross shared memory between the
//   coalesced order and the chunks' (lsx_pad keeps that free of conflicts).
//   y lines: a block takes up to 8 neighbouring columns, a whole 32-byte
//   sector of each row, times the chunks of a line; lines of more than 32
//   chunks (512 rows) are shared by a cluster of 2, 4 or 8 blocks.  The
//   reduced rows of a column go to one block of the cluster through
//   distributed shared memory (each block owns 8 / nc of the columns), are
//   solved there and come back.
// The reduced system (2P rows of a line, at most 512 rows per block: a chunk's
// pair per thread) is solved by parallel cyclic reduction with the multipliers
// that the factorisation left (pcr_factor), staged in shared memory at the
// start.
// REM: the line's length is no multiple of LSF_M.  Its last chunk has up to
// 31 rows, whose rows past the 16th belong to a thread of their own; the two
// hand the sweeps' running value to each other through shared memory.  All
// threads then sweep 16 rows without a test: the constants of a chunk's first
// and last row (fac_a_body) and the zeros beside them pass those rows by, and
// a remainder thread repeats its last row's.
// What bounds it is memory latency (16 warps to an SM at 128 registers), so
// the loads of a phase are issued together (ld_now).  The operations and
// their order are those of k_sol_a .. k_resid, which the other lines take, so
// that the results are the same bit for bit.
// Measured with the two early-exit factor launches (us, before -> after; x
// took one 256-thread block per line, y seven kernels moving 95 B per cell):
// 2048 x 2048 x 119 -> 75, y 138 -> 94; 4096 x 4096 x 1160 -> 247, y 424 ->
// 330; 250 x 500 x 28 -> 20, y 72 -> 25 (the 20-row last chunks walked global
// memory); 1024 x 1024 x 41 -> 23, y 51 -> 29.
// ---------------------------------------------------------------------------
constexpr int LSF_T = 256;     // most threads of a block
constexpr int LSF_COLS = 8;    // columns of a y block
struct LsfShape {
    int nline;  // lines of a block
    int nch;    // threads of a line in a block (its chunks, and the remainder rows' thread)
    int slots;  // lines whose reduced rows a block solves
    int nc;     // blocks of a cluster
    int nblk;   // blocks of the grid
    int nt;     // threads of a block: its lines' chunks, in whole warps
};

// the address of a shared-memory word of this block in block `rank` of the cluster
__device__ __forceinline__ float *cluster_peer(float *p, int rank) {
    uint64_t q;
    asm("mapa.u64 %0, %1, %2;" : "=l"(q) : "l"(p), "r"(rank));
    return reinterpret_cast<float *>(q);
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// a read-only load that stays where it is written, ahead of later barriers
__device__ __forceinline__ float ld_now(const float *p) {
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
// 16 bytes to shared memory without a register, and the wait for all of them
__device__ __forceinline__ void copy16_async(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// shared memory of a block, in floats: the reduction's multipliers, the
// reduced right-hand sides twice, the solved pairs of the block's chunks with
// a neighbour on either side, the remainder rows' exchange and, for x, the
// staged lines
static size_t lsf_smem_floats(int dir, const LinePart &lp, const LsfShape &S) {
    return (size_t)S.slots * pcr_words(lp) + (size_t)2 * S.slots * 2 * lp.P + (size_t)S.nline * (2 * S.nch + 4) +
           (size_t)4 * S.nline + (dir == 0 ? (size_t)S.nline * (lsx_pad(lp.L) + 1) : 0);
}

template <typename T, int DIR, bool PER, bool REM>
__global__ void __launch_bounds__(LSF_T, 2) k_linesolve(Grid g, Fields<T> f, LinePart lp, LsfShape S, int clear_dirty) {
    extern __shared__ __align__(16) float shf[];
    constexpr int M = LSF_M;
    const int P = lp.P, L = lp.L, n = 2 * P, tid = threadIdx.x, NT = blockDim.x;
    const int PT = P + (REM ? 1 : 0);  // threads of a line
    const bool clus = DIR == 1 && S.nc > 1;
    if (clus) cluster_arrive();  // every block of the cluster has started before the first remote store
    const int rank = clus ? (int)(blockIdx.x % (unsigned)S.nc) : 0;
    const int grp = clus ? (int)(blockIdx.x / (unsigned)S.nc) : (int)blockIdx.x;
    // the factorisation of this stage is complete: the MASK9 change flag
    // can be reset for UPDATE_MASK to set again
    if (clear_dirty && blockIdx.x == 0 && tid == 0) *f.m9_dirty = 0;
    const int nred = S.slots * n, steps = pcr_steps(n), n4 = (n + 3) & ~3, pw = pcr_words(lp);
    float *MUL = shf;                  // [slots][pw]
    float *R0 = MUL + S.slots * pw, *R1 = R0 + nred;
    const int rw = 2 * S.nch + 4;
    float *res = R1 + nred;            // per line: -, left neighbour, the chunks' pairs, right neighbour, -
    float *ex = res + S.nline * rw;    // [4][nline]
    float *stage = ex + 4 * S.nline;   // x: the block's lines
    const int SW = lsx_pad(L) + 1;

    // this thread's line and chunk (y: consecutive threads on consecutive columns)
    const int ln = DIR == 0 ? tid / PT : tid % S.nline;
    const int cl = DIR == 0 ? tid - ln * PT : tid / S.nline;
    const int ct = rank * S.nch + cl;       // chunk, or P: the remainder rows of chunk P-1
    // x: a block's lines from grp*nline; y: its columns from nline*grp of the
    // plane (sector-aligned), of which the interior ones are lines
    const int l0 = grp * S.nline - (DIR == 0 ? 0 : g.ib), l = l0 + ln;
    const bool on = ln < S.nline && cl < S.nch && ct < PT && l >= 0 && l < lp.nlines;
    const bool rem = REM && on && ct == P, last = REM && on && ct == P - 1;
    const int ch = rem ? P - 1 : ct;
    const int s = ct * M, nr = rem ? L - s : M;   // this thread's first row and its rows
    constexpr int K0 = REM ? 0 : 1, K1 = REM ? M : M - 1;  // rows that the sweeps walk
    const int fst = DIR == 0 ? (rem ? 1 : P) : g.pitch;
    // offset of row k's factors from the first row's (of the last row for the
    // rows that a remainder does not have: loaded, never used)
#define LSF_OFF(k) ((REM ? min((k), nr - 1) : (k)) * fst)
    const size_t fq = on ? fac_at<DIR>(g, lp, l, s) : 0;

    // the multipliers, in flight until the first reduction
    for (int q = tid; q < S.slots * (pw / 4); q += NT) {
        const int slot = q / (pw / 4);
        const int rl = DIR == 0 ? l0 + slot : l0 + slot * S.nc + rank;
        if (rl >= 0 && rl < lp.nlines) copy16_async(MUL + 4 * q, pcr_line<T, DIR>(f, lp, rl) + 4 * (q - slot * (pw / 4)));
    }
    // the right-hand side (x: staged below), normalised, and the sweeps' constants
    float d[M], y[M], x0[M], av[M], lv[M], cv[M];
    if (on) {
        const float *IT = f.fac_it[DIR] + fq, *FA = f.fac_A[DIR] + fq, *LR = f.fac_lr[DIR] + fq, *CP = f.fac_cp[DIR] + fq;
#pragma unroll
        for (int k = 0; k < M; k++) {
            if (DIR == 1) d[k] = ld_now((const float *)f.rhs_y + fq + LSF_OFF(k));
            x0[k] = ld_now(IT + LSF_OFF(k));
        }
#pragma unroll
        for (int k = K0; k < K1; k++) {
            av[k] = ld_now(FA + LSF_OFF(k));
            lv[k] = ld_now(LR + LSF_OFF(k));
            cv[k] = ld_now(CP + LSF_OFF(k));
        }
    }
    float cs = 0.0f, ae = 0.0f, sc0 = 1.0f, sc1 = 1.0f;
    if (on) {
        const FacLine fl = fac_line(f.fac_red[DIR], lp, l);
        cs = ld_now(fl.cs + ch);
        ae = ld_now(fl.ae + ch);
        if (PER) {
            if (ch == 0) sc0 = 1.0f / (1.0f + ld_now(fl.tail + 0));      // row 0: d / (1 + c_end)
            if (ch == P - 1) sc1 = 1.0f / (1.0f + ld_now(fl.tail + 1));  // row L-1: d / (1 + a_beg)
        }
    }
    if (DIR == 0) {
        const int nl = min(S.nline, lp.nlines - l0);
        for (int q = 0; q < nl; q++) {
            const T *src = f.rhs_x + (size_t)(g.jb + l0 + q) * g.pitch + g.ib;
#pragma unroll 4
            for (int k = tid; k < L; k += NT) stage[q * SW + lsx_pad(k)] = (float)ro(src + k);
        }
        __syncthreads();
    }
    if (on) {
#pragma unroll
        for (int k = 0; k < M; k++)
            d[k] = __fmul_rn(DIR == 0 ? stage[ln * SW + lsx_pad(s + (REM ? min(k, nr - 1) : k))] : d[k], x0[k]);
    }
    // the reduced rows this thread solves: the pair of chunk rc of line rl (slot rsl)
    const int rsl = tid / P, rc = tid - rsl * P;
    const int rl = DIR == 0 ? l0 + rsl : l0 + rsl * S.nc + rank;
    const bool ron = rsl < S.slots && rl >= 0 && rl < lp.nlines;

#pragma unroll
    for (int pass = 0; pass < 2; pass++) {
        // the chunk's forward and backward sweep
        auto forward = [&](float yp) {
#pragma unroll
            for (int k = K0; k < K1; k++) {
                yp = __fmaf_rn(d[k], av[k], -__fmul_rn(lv[k], yp));  // rounded as in k_sol_a
                y[k] = yp;
            }
            return yp;
        };
        auto backward = [&](float yn) {
#pragma unroll
            for (int k = K1 - 1; k >= K0; k--) {
                yn = __fmaf_rn(-cv[k], yn, y[k]);
                y[k] = yn;
            }
            return yn;
        };
        float rs = 0.0f, re = 0.0f, yn = 0.0f;
        if (on && !rem) {
            const float yp = forward(0.0f);
            if (last) ex[ln] = yp;
        }
        if (REM) {
            // the last chunk: forward through both of its threads, then back
            __syncthreads();
            if (rem) {
                const float yp = ex[ln];
                forward(yp);
                ex[S.nline + ln] = backward(0.0f);
                float de = d[0], ye = yp;  // d of the chunk's last row, y of the one before
#pragma unroll
                for (int k = 1; k < M; k++)
                    if (k == nr - 1) {
                        de = d[k];
                        ye = y[k - 1];
                    }
                ex[2 * S.nline + ln] = ye;
                ex[3 * S.nline + ln] = __fmul_rn(de, sc1);
            }
            __syncthreads();
            if (last) yn = ex[S.nline + ln];
        }
        if (on && !rem) {
            backward(yn);
            rs = __fmul_rn(d[0], sc0) - cs * y[1];
            re = REM && last ? ex[3 * S.nline + ln] - ae * ex[2 * S.nline + ln]
                             : __fmul_rn(d[M - 1], sc1) - ae * y[M - 2];
        }
        if (clus && pass == 0) cluster_wait();
        if (on && !rem) {
            // the reduced right-hand sides, to the block that solves this line
            float *dst = R0 + (DIR == 0 ? ln : ln / S.nc) * n + 2 * ch;
            if (clus) dst = cluster_peer(dst, ln % S.nc);
            dst[0] = rs;
            dst[1] = re;
        }
        if (on) {
            // the reconstruction's constants arrive while the reduced system is solved
            const float *PP = f.fac_p[DIR] + fq, *QQ = f.fac_q[DIR] + fq;
#pragma unroll
            for (int k = K0; k < K1; k++) {
                av[k] = ld_now(PP + LSF_OFF(k));
                lv[k] = ld_now(QQ + LSF_OFF(k));
            }
        }
        if (pass == 0) copies_wait();
        if (clus) {
            cluster_arrive();
            cluster_wait();
        } else {
            __syncthreads();
        }
        // parallel cyclic reduction
        float *r = R0 + 2 * tid, *r2 = R1 + 2 * tid;
        const float *m = MUL + rsl * pw + 2 * rc;
        float2 rr = make_float2(0.0f, 0.0f);
        if (ron) {
            rr = *(const float2 *)r;
            // neighbours one row away: a pair's rows are each other's
            const float2 a = *(const float2 *)m, b = *(const float2 *)(m + n4);
            float x = rr.x, y_ = rr.y;
            if (rc > 0) x += a.x * r[-1];
            x += b.x * rr.y;
            y_ += a.y * rr.x;
            if (rc < P - 1) y_ += b.y * r[2];
            rr = make_float2(x, y_);
            *(float2 *)r2 = rr;
        }
        __syncthreads();
        for (int st = 1; st < steps; st++) {
            float *t = r;
            r = r2;
            r2 = t;
            m += 2 * n4;
            if (ron) {
                // whole pairs: 2^st rows are 2^(st-1) chunks
                const int dist = 1 << st, dc = dist >> 1;
                const float2 a = *(const float2 *)m, b = *(const float2 *)(m + n4);
                if (rc >= dc) {
                    const float2 v = *(const float2 *)(r - dist);
                    rr.x += a.x * v.x;
                    rr.y += a.y * v.y;
                }
                if (rc + dc < P) {
                    const float2 v = *(const float2 *)(r + dist);
                    rr.x += b.x * v.x;
                    rr.y += b.y * v.y;
                }
                *(float2 *)r2 = rr;
            }
            __syncthreads();
        }
        if (ron) {
            const float2 di = *(const float2 *)(m + 2 * n4);
            rr = make_float2(rr.x / di.x, rr.y / di.y);
        }
        if (PER) {  // Sherman-Morrison with both ends of the line's solution
            if (ron && rc == 0) r[0] = rr.x;
            if (ron && rc == P - 1) r[1] = rr.y;
            __syncthreads();
            if (ron) {
                const FacLine fl = fac_line(f.fac_red[DIR], lp, rl);
                const float *z = r - 2 * rc;
                const float beta = (ro(fl.tail + 0) * z[0] - ro(fl.tail + 1) * z[n - 1]) / ro(fl.tail + 2);
                rr.x = rr.x + beta * ro(fl.x2 + 2 * rc);
                rr.y = rr.y + beta * ro(fl.x2 + 2 * rc + 1);
            }
        }
        if (ron) {
            // to the chunk's own pair and, at the end of a block's chunks (or
            // of a periodic line), to the neighbour's outer place
            const int q = clus ? rc / S.nch : 0, cq = rc - q * S.nch;
            float *own = res + (DIR == 0 ? rsl : rsl * S.nc + rank) * rw;
            auto at = [&](int blk, int pos) { return clus ? cluster_peer(own + pos, blk) : own + pos; };
            *(float2 *)at(q, 2 + 2 * cq) = rr;
            if (clus && rc < P - 1 && cq == S.nch - 1) *at(q + 1, 1) = rr.y;
            if (clus && rc > 0 && cq == 0) *at(q - 1, 2 + 2 * S.nch) = rr.x;
            if (PER && rc == P - 1) *at(0, 1) = rr.y;
            if (PER && rc == 0) {
                const int ql = clus ? (P - 1) / S.nch : 0;
                *at(ql, 2 + 2 * (P - ql * S.nch)) = rr.x;
            }
        }
        if (clus) {
            cluster_arrive();
            cluster_wait();
        } else {
            __syncthreads();
        }
        // reconstruction; after the first pass the residual in d's place
        const float *rv = res + ln * rw + 2 + 2 * (ch - rank * S.nch);
        const float xs = on ? rv[0] : 0.0f, xe = on ? rv[1] : 0.0f;
        float xl = on && (PER || ch > 0) ? rv[-1] : 0.0f, xr = on && (PER || ch < P - 1) ? rv[2] : 0.0f;
        if (on) {
#pragma unroll
            for (int k = K0; k < K1; k++) y[k] = y[k] - av[k] * xs - lv[k] * xe;
            if (!rem) y[0] = xs;
            if (!REM || !(rem || last)) y[M - 1] = xe;
            if (REM) {
#pragma unroll
                for (int k = 0; k < M; k++)
                    if (rem && k >= nr - 1) y[k] = xe;
            }
        }
        if (REM && pass == 0) {
            // the last chunk's two threads are each other's neighbours
            if (last) ex[2 * S.nline + ln] = y[M - 1];
            if (rem) ex[3 * S.nline + ln] = y[0];
            __syncthreads();
            if (rem) xl = ex[2 * S.nline + ln];
            if (last) xr = ex[3 * S.nline + ln];
        }
        if (on) {
            if (pass == 0) {
                const float *AH = f.fac_ah[DIR] + fq, *AL = f.fac_al[DIR] + fq, *CH = f.fac_ch[DIR] + fq,
                            *CL = f.fac_cl[DIR] + fq;
                // rows whose coefficients are loaded together
                constexpr int HB = 8;
#pragma unroll
                for (int k0 = 0; k0 < M; k0 += HB) {
                    float ah[HB], al[HB], ch_[HB], cl_[HB];
#pragma unroll
                    for (int q = 0; q < HB; q++) {
                        ah[q] = ld_now(AH + LSF_OFF(k0 + q));
                        al[q] = ld_now(AL + LSF_OFF(k0 + q));
                        ch_[q] = ld_now(CH + LSF_OFF(k0 + q));
                        cl_[q] = ld_now(CL + LSF_OFF(k0 + q));
                    }
#pragma unroll
                    for (int q = 0; q < HB; q++) {
                        const int k = k0 + q;
                        const float xm = k > 0 ? y[k > 0 ? k - 1 : 0] : xl;
                        const float xp = k < M - 1 && (!REM || k < nr - 1) ? y[k < M - 1 ? k + 1 : k] : xr;
                        d[k] = residual(d[k], y[k], xm, xp, ah[q], al[q], ch_[q], cl_[q]);
                        x0[k] = y[k];
                    }
                }
                // the sweeps' constants again (L2)
                const float *FA = f.fac_A[DIR] + fq, *LR = f.fac_lr[DIR] + fq, *CP = f.fac_cp[DIR] + fq;
#pragma unroll
                for (int k = K0; k < K1; k++) {
                    av[k] = ld_now(FA + LSF_OFF(k));
                    lv[k] = ld_now(LR + LSF_OFF(k));
                    cv[k] = ld_now(CP + LSF_OFF(k));
                }
            } else {
#pragma unroll
                for (int k = 0; k < M; k++)
                    if (!REM || k < nr) {
                        const float x = x0[k] + y[k];
                        if (DIR == 0) stage[ln * SW + lsx_pad(s + k)] = x;
                        else f.V[fq + (size_t)k * fst] = (T)x;
                    }
            }
        }
    }
#undef LSF_OFF
    if (DIR == 0) {
        __syncthreads();
        const int nl = min(S.nline, lp.nlines - l0);
        for (int q = 0; q < nl; q++) {
            T *dst = f.U + (size_t)(g.jb + l0 + q) * g.pitch + g.ib;
            for (int k = tid; k < L; k += NT) dst[k] = (T)stage[q * SW + lsx_pad(k)];
        }
    }
}

// ---------------------------------------------------------------------------
// GET_Eta_U_V_HU_HV tail (etauv_solver.F:558-600): dry zeroing, HU/HV and
// the Froude cap, with the MASK of the start of the stage.
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void post_cell(const Grid &g, const Fields<T> &f, int i, int j) {
    const int id = IDI(i, j);
    const T mdf = GC(min_depth_frc);
    const bool interior = !(i < g.ib || i > g.ie || j < g.jb || j > g.je);
    if (interior) {
        if (!g.dispersion) {
            const T Hm = tmax(ro(f.H + (id)), mdf);
            f.U[id] = f.Ubar[id] / Hm;
            f.V[id] = f.Vbar[id] / Hm;
        }
        if (ro(f.MASK + (id)) < 1) {
            f.Ubar[id] = (T)0;
            f.Vbar[id] = (T)0;
            f.U[id] = (T)0;
            f.V[id] = (T)0;
            f.HU[id] = (T)0;
            f.HV[id] = (T)0;
        } else {
            const T Hm = tmax(ro(f.H + (id)), mdf);
            const T u = f.U[id], v = f.V[id];
            f.HU[id] = Hm * u;
            f.HV[id] = Hm * v;
            const T Utotal = fsqrt(u * u + v * v);
            const T Fr = fsqrt((T)GRAV * Hm);
            if (Utotal / Fr > GC(froude_cap)) {
                const T th = fatan2(v, u);
                const T un = GC(froude_cap) * Fr * fcos(th);
                const T vn = GC(froude_cap) * Fr * fsin(th);
                f.U[id] = un;
                f.V[id] = vn;
                f.HU[id] = un * Hm;
                f.HV[id] = vn * Hm;
            }
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(256) k_post(Grid g, Fields<T> f) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= g.Mloc || j >= g.Nloc) return;
    post_cell(g, f, i, j);
}

// Ubar = HU, Vbar = HV on every cell when DISPERSION is off (etauv_solver.F:596-600)
template <typename T>
__global__ void k_nodisp_copy(Grid g, Fields<T> f) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= g.Mloc || j >= g.Nloc) return;
    const int id = IDI(i, j);
    f.Ubar[id] = f.HU[id];
    f.Vbar[id] = f.HV[id];
}

// ---------------------------------------------------------------------------
// UPDATE_MASK (masks.F:51-205): MASK (Jacobi into MASKn), the Depthx/
// Depthy reset at old-dry cells, MASK9.  Launched over (Mloc+1) x (Nloc+1)
// so that every face has a thread.
// ---------------------------------------------------------------------------
// The sign of eta + h, with h the Depth as given in double (the FP64
// build's own Depth, the mixed build's double copy of it): +1 for
// eta > -h, -1 for eta < -h, 0 for equality, as the double comparisons of
// masks.F:107, 129 decide.  The mixed build decides in float where the
// float sum's margin exceeds its rounding (about 2 ulps of the larger term,
// plus the rounding of the stored float Depth), which gives the same sign,
// and evaluates the rest in double: FP64 instructions run only at cells
// within a few ulps of the threshold.
__device__ __forceinline__ int wet_test(double eta, double hf, const double *) {
    return eta > -hf ? 1 : (eta < -hf ? -1 : 0);
}
// the double comparison, out of line so that the float path of the callers
// keeps its registers
static __device__ __noinline__ int wet_test_double(float eta, const double *hdp) {
    const double e = (double)eta, hd = *hdp;
    return e > -hd ? 1 : (e < -hd ? -1 : 0);
}
__device__ __forceinline__ int wet_test(float eta, float hf, const double *hdp) {
    const float s = eta + hf;
    const float tol = 4.0e-7f * fmaxf(fabsf(eta), fabsf(hf)) + 1.0e-30f;
    if (s > tol) return 1;
    if (s < -tol) return -1;
    return wet_test_double(eta, hdp);  // the double depth only here
}

template <typename T>
__device__ __forceinline__ bool in_mask_range(const Grid &g, int a, int b) {
    return a >= g.ib - 2 && a <= g.ie + 2 && b >= g.jb - 2 && b <= g.je + 2;
}
template <typename T>
__device__ __forceinline__ int new_mask(const Grid &g, const Fields<T> &f, int a, int b) {
    const size_t q = IDI(a, b);
    const int m = ro(f.MASK + (q));
    if (!in_mask_range<T>(g, a, b) || ro(f.MASK_STRUC + (q)) != 1) return m;
    // total-depth tests (masks.F:107, 129) of eta against Depth as given, in
    // double (wet_test)
    const T eta = ro(f.Eta + (q));
    const int side = wet_test(eta, ro(f.Depth + (q)), f.DepthD + q);
    if (m < 1) {
        int r = m;
        if (side > 0) r = 1;
        if (ro(f.MASK + (IDI(a - 1, b))) == 1 && ro(f.Eta + (IDI(a - 1, b))) > eta) r = 1;
        if (ro(f.MASK + (IDI(a + 1, b))) == 1 && ro(f.Eta + (IDI(a + 1, b))) > eta) r = 1;
        if (ro(f.MASK + (IDI(a, b - 1))) == 1 && ro(f.Eta + (IDI(a, b - 1))) > eta) r = 1;
        if (ro(f.MASK + (IDI(a, b + 1))) == 1 && ro(f.Eta + (IDI(a, b + 1))) > eta) r = 1;
        return r;
    }
    return (side < 0) ? 0 : m;
}

// one thread of UPDATE_MASK at (i, j) in 0..Mloc x 0..Nloc
template <typename T>
__device__ __forceinline__ void mask_cell(const Grid &g, const Fields<T> &f, int i, int j) {
    // Depthx at x-face i of row j
    if (j < g.Nloc && j >= g.jb - 2 && j <= g.je + 2) {
        const bool rin = (i >= g.ib - 2 && i <= g.ie + 2);
        const bool lin = (i - 1 >= g.ib - 2 && i - 1 <= g.ie + 2);
        if (rin && ro(f.MASK + (IDI(i, j))) < 1) f.Depthx[IDI(i, j)] = ro(f.Depth + (IDI(i - 1, j)));
        else if (lin && ro(f.MASK + (IDI(i - 1, j))) < 1) f.Depthx[IDI(i, j)] = ro(f.Depth + (IDI(i, j)));
    }
    // Depthy at y-face j of column i
    if (i < g.Mloc && i >= g.ib - 2 && i <= g.ie + 2) {
        const bool tin = (j >= g.jb - 2 && j <= g.je + 2);
        const bool bin = (j - 1 >= g.jb - 2 && j - 1 <= g.je + 2);
        if (tin && ro(f.MASK + (IDI(i, j))) < 1) f.Depthy[IDI(i, j)] = ro(f.Depth + (IDI(i, j - 1)));
        else if (bin && ro(f.MASK + (IDI(i, j - 1))) < 1) f.Depthy[IDI(i, j)] = ro(f.Depth + (IDI(i, j)));
    }
    if (i >= g.Mloc || j >= g.Nloc) return;
    const int id = IDI(i, j);
    f.MASKn[id] = (uint8_t)new_mask(g, f, i, j);
    // MASK9 on Ibeg-1..Iend+1 x Jbeg-1..Jend+1; 0 elsewhere (never written
    // in the reference, whose temporary is fresh memory)
    uint8_t m9 = 0;
    if (i >= g.ib - 1 && i <= g.ie + 1 && j >= g.jb - 1 && j <= g.je + 1) {
        if (g.visc_breaking) {
            m9 = 1;
        } else {
            int p = 1;
            for (int b = -1; b <= 1; b++)
                for (int a = -1; a <= 1; a++) p *= new_mask(g, f, i + a, j + b);
            if (fabs_(ro(f.Eta + (id))) / tmax(ro(f.Depth + (id)), GC(min_depth_frc)) > GC(swe_eta_dep)) p = 0;
            m9 = (uint8_t)p;
        }
    }
    if (f.MASK9[id] != m9) *f.m9_dirty = 1;  // the tridiagonal matrices change
    f.MASK9[id] = m9;
}

template <typename T>
__global__ void __launch_bounds__(256) k_mask(Grid g, Fields<T> f) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i > g.Mloc || j > g.Nloc) return;
    mask_cell(g, f, i, j);
}

// ---------------------------------------------------------------------------
// BREAKING (breaker.F:87-353), default branch
// ---------------------------------------------------------------------------
template <typename T> struct BrkLocal {
    T tmp1, tmp2, tmp3, et;
};
template <typename T>
__device__ __forceinline__ BrkLocal<T> brk_local(const Grid &g, const Fields<T> &f, int id) {
    BrkLocal<T> b;
    b.tmp3 = fsqrt((T)GRAV * tmax(GC(min_depth_frc), ro(f.H + (id))));
    b.tmp1 = GC(cbrk1) * b.tmp3;
    b.tmp2 = GC(cbrk2) * b.tmp3;
    b.et = ro(f.ETAT + (id));
    return b;
}
template <typename T>
__device__ __forceinline__ bool in_wk_zone(const Grid &g, int i, int j) {
    const T xmk = i2r<T>(i - g.ib) * GC(DX), ymk = i2r<T>(j - g.jb) * GC(DY);
    return fabs_(xmk - GC(xc_wk)) < GC(width_wk) && fabs_(ymk - GC(yc_wk)) < GC(ywidth_wk) / (T)2;
}
template <typename T>
__device__ __forceinline__ T nu_of(const Grid &g, const BrkLocal<T> &b, T age, bool zone, T depth, T eta) {
    const T mdf = GC(min_depth_frc);
    if (zone) {
        if (b.et > tmin(b.tmp2, GC(wavemaker_cbrk) * b.tmp3)) {
            const T cap1 = (T)1 * (tmax(depth, mdf) + eta);
            return cap1 * GC(wavemaker_cbrk) * b.tmp3 + GC(nu_bkg);
        }
        return (T)0 + GC(nu_bkg);
    }
    if (age > (T)0 && age < GC(T_brk) && b.et > b.tmp2) {
        const T cap1 = (T)1 * (tmax(depth, mdf) + eta);
        return cap1 * b.tmp2 + GC(nu_bkg);
    }
    return (T)0 + GC(nu_bkg);
}
template <typename T>
__device__ __forceinline__ T nu_value(const Grid &g, const Fields<T> &f, int id, const BrkLocal<T> &b, T age,
                                      bool zone) {
    return nu_of(g, b, age, zone, ro(f.Depth + (id)), ro(f.Eta + (id)));
}

// roller flux and undertow of a breaking cell (breaker.F:316-339):
// C1 = max(|ETAt|/tmp4, sqrt(g|H|)), R = min(|0.45 ETAt/max(C1,SMALL)|,
// 0.1638), ROLLER = |C1 - |u|| R (eta - ETAmean), UNDERTOW = -ROLLER times
// the direction cosines of ANGLE; 0.45 is a default-REAL literal and 0.1638
// a _SP one, so both enter FP64 as their float values.  ETAmean is zero
// until a mean is computed.
template <typename T>
__device__ __forceinline__ void roller_cell(const Grid &g, const Fields<T> &f, int id, T et) {
    const T ex = ro(f.ETAx + (id)), ey = ro(f.ETAy + (id));
    const T tmp4 = tmax(fsqrt(ex * ex + ey * ey), (T)SMALL);
    const T ANGLE = fatan2(-ey, -ex) * (T)180 / (T)PI_SP;
    const T C1 = tmax(fabs_(et) / tmp4, fsqrt((T)GRAV * fabs_(ro(f.H + (id)))));
    T R = fabs_((T)(double)0.45f * et / tmax(C1, (T)SMALL));
    R = tmin(R, (T)(double)0.1638f);
    const T u = f.U[id], v = f.V[id];
    const T em = g.stats ? f.ETAmean[id] : (T)0;
    const T rf = fabs_(C1 - fsqrt(u * u + v * v)) * R * (ro(f.Eta + (id)) - em);
    f.ROLLER[id] = rf;
    f.UNDERTOW_U[id] = -rf * fcos(ANGLE * (T)PI_SP / (T)180);
    f.UNDERTOW_V[id] = -rf * fsin(ANGLE * (T)PI_SP / (T)180);
}

// the breaking branch of the viscosity (outside the wavemaker zone)
template <typename T> __device__ __forceinline__ bool breaking_now(const Grid &g, const BrkLocal<T> &b, T age) {
    return age > (T)0 && age < GC(T_brk) && b.et > b.tmp2;
}

// A stage adds a cell at most once, and its sweep empties the list.  Launched
// again without the sweep (fw_time_kernel, fw_autotune) cells come again; those
// past the list's end are left out.
template <typename T> __device__ __forceinline__ void add_cand(const Grid &g, const Fields<T> &f, int id) {
    const unsigned slot = (unsigned)atomicAdd(f.ncand, 1);
    if (slot < (unsigned)cand_cap(g)) f.cand[slot] = id;
}

template <typename T>
__device__ __forceinline__ void break_cell(const Grid &g, const Fields<T> &f, int i, int j) {
    const int id = IDI(i, j);
    const T age = ro(f.AGE + (id));
    if (i < g.ib - 1 || i > g.ie + 1 || j < g.jb - 1 || j > g.je + 1) {
        f.AGEn[id] = age;
        return;
    }
    const T DT = DTV;
    const BrkLocal<T> b = brk_local(g, f, id);
    T an = age;
    bool cand = false;
    if (b.et >= b.tmp1 && (age == (T)0 || age > GC(T_brk))) an = DT;
    else if (age > (T)0) an = age + DT;
    else if (b.et >= b.tmp2) cand = true;
    f.AGEn[id] = an;
    const bool zone = in_wk_zone<T>(g, i, j);
    if (cand) add_cand(g, f, id);
    if (zone || !cand) f.nu[id] = nu_value(g, f, id, b, an, zone);
    if (g.track_roller && !zone && !cand && breaking_now(g, b, an)) roller_cell(g, f, id, b.et);
}

template <typename T>
__global__ void __launch_bounds__(256) k_break_a(Grid g, Fields<T> f) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= g.Mloc || j >= g.Nloc) return;
    break_cell(g, f, i, j);
}

// The stage's GET_Eta_U_V_HU_HV tail, UPDATE_MASK and the parallel part of
// BREAKING in one pass: each reads only values that are final before it
// starts (U, V from the line solves; Eta, H from ESTIMATE_HUV; the MASK of
// the start of the stage; AGE of the previous stage) and writes disjoint
// arrays, so one thread can do all three.  Launched over (Mloc+1) x (Nloc+1).
// A cell of the interior that is wet, with wet cells to its west and south
// and viscosity breaking on (MASK9 = 1), needs one value of each input: they
// are loaded together before the first use (the parts one after the other,
// each loading behind the stores of the one before: 88 us at 2048 x 2048, now
// 52 with 32-bit offsets and lines ahead, 1.5 times the floor of its 57 B per
// cell).  The others take the parts one by one.
template <typename T>
__global__ void __launch_bounds__(256) k_post_mask_break(Grid g, Fields<T> f, Ahead ah) {
    prefetch_ahead<T>(g, ah, blockIdx.y, 0);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i > g.Mloc || j > g.Nloc) return;
    const bool in = i >= g.ib && i <= g.ie && j >= g.jb && j <= g.je;
    if (in && g.visc_breaking && g.dispersion) {
        const int id = i + j * g.pitch;
        const int m = ro(f.MASK, id), mw = ro(f.MASK, id - 1), ms = ro(f.MASK, id - g.pitch),
                  st = ro(f.MASK_STRUC, id), m9 = f.MASK9[id];
        const T h = ro(f.H, id), u = f.U[id], v = f.V[id], age = ro(f.AGE, id), eta = ro(f.Eta, id), dep = ro(f.Depth, id);
        BrkLocal<T> b;
        b.et = ro(f.ETAT, id);
        const T mdf = GC(min_depth_frc);
        if (m >= 1 && mw >= 1 && ms >= 1) {
            // GET_Eta_U_V_HU_HV tail (post_cell)
            const T Hm = tmax(h, mdf);
            f.HU[id] = Hm * u;
            f.HV[id] = Hm * v;
            const T Utotal = fsqrt(u * u + v * v);
            const T Fr = fsqrt((T)GRAV * Hm);
            // (a ratio of at most 1 does not exceed a cap of at least 1)
            if (!(Utotal <= Fr && GC(froude_cap) >= (T)1) && Utotal / Fr > GC(froude_cap)) {
                const T th = fatan2(v, u);
                const T un = GC(froude_cap) * Fr * fcos(th);
                const T vn = GC(froude_cap) * Fr * fsin(th);
                f.U[id] = un;
                f.V[id] = vn;
                f.HU[id] = un * Hm;
                f.HV[id] = vn * Hm;
            }
            // BREAKING (break_cell)
            b.tmp3 = h == h ? Fr : h;  // sqrt(g max(mdf, h)), NaN where h is
            b.tmp1 = GC(cbrk1) * b.tmp3;
            b.tmp2 = GC(cbrk2) * b.tmp3;
            const T DT = DTV;
            T an = age;
            bool cand = false;
            if (b.et >= b.tmp1 && (age == (T)0 || age > GC(T_brk))) an = DT;
            else if (age > (T)0) an = age + DT;
            else if (b.et >= b.tmp2) cand = true;
            f.AGEn[id] = an;
            const bool zone = in_wk_zone<T>(g, i, j);
            if (cand) add_cand(g, f, id);
            if (zone || !cand) f.nu[id] = nu_of(g, b, an, zone, dep, eta);
            if (g.track_roller && !zone && !cand && breaking_now(g, b, an)) roller_cell(g, f, id, b.et);
            // UPDATE_MASK (mask_cell; wet cells beside it: no depth reset)
            f.MASKn[id] = (uint8_t)(st == 1 && wet_test(eta, dep, f.DepthD + id) < 0 ? 0 : m);
            if (m9 != 1) {
                *f.m9_dirty = 1;  // the tridiagonal matrices change
                f.MASK9[id] = 1;
            }
            return;
        }
    }
    if (i < g.Mloc && j < g.Nloc) {
        post_cell(g, f, i, j);
        break_cell(g, f, i, j);
    }
    mask_cell(g, f, i, j);
}

// the neighbour test of one candidate (breaker.F:182-224); N = new values
template <typename T>
__device__ __forceinline__ bool brk_neigh(const Grid &g, const Fields<T> &f, const volatile T *N, int i, int j,
                                          T DT) {
    const size_t id = IDX(i, j);
    const T ex = ro(f.ETAx + (id)), ey = ro(f.ETAy + (id));
    const T ANGLE = fatan2(-ey, -ex) * (T)180 / (T)PI_SP;
    const T tmp4 = tmax(fsqrt(ex * ex + ey * ey), (T)SMALL);
    const T Hc = ro(f.H + (id));
    const T C = tmin(fabs_(ro(f.ETAT + (id))) / tmp4, fsqrt((T)GRAV * fabs_(Hc)));
    const T DX = GC(DX), DY = GC(DY);
    const T propxy = fsqrt(DX * DX + DY * DY) / tmax(C, (T)SMALL);
    const T propx = fsqrt(DX * DX) / tmax(C, (T)SMALL);
    const T propy = fsqrt(DY * DY) / tmax(C, (T)SMALL);
    const T *O = f.AGE;  // values before the sweep
#define NW(a, b) N[IDX(i + (a), j + (b))]
#define OL(a, b) O[IDX(i + (a), j + (b))]
    bool hit = false;
    T A1, A2, A3;
    if (ANGLE >= (T)0 && ANGLE < (T)90) {
        A1 = NW(-1, 0);
        A2 = NW(-1, -1);
        A3 = NW(0, -1);
        if ((A1 >= DT && A1 > propx) || (A2 >= DT && A2 > propxy) || (A3 >= DT && A3 > propy)) hit = true;
    }
    if (ANGLE >= (T)90 && ANGLE < (T)180) {
        A1 = OL(1, 0);
        A2 = NW(1, -1);
        A3 = NW(0, -1);
        if ((A1 >= DT && A1 > propx) || (A2 >= DT && A2 > propxy) || (A3 >= DT && A3 > propy)) hit = true;
    }
    if (ANGLE >= (T)-180 && ANGLE < (T)-90) {
        A1 = OL(1, 0);
        A2 = OL(1, 1);
        A3 = OL(0, 1);
        if ((A1 >= DT && A1 > propx) || (A2 >= DT && A2 > propxy) || (A3 >= DT && A3 > propy)) hit = true;
    }
    if (ANGLE >= (T)-90 && ANGLE < (T)0) {
        A1 = OL(0, 1);
        A2 = OL(-1, 1);
        A3 = NW(-1, 0);
        if ((A1 >= DT && A1 > propy) || (A2 >= DT && A2 > propxy) || (A3 >= DT && A3 > propx)) hit = true;
    }
#undef NW
#undef OL
    return hit;
}

// one candidate of the sweep: 0 -> DT when a neighbour before it carries
// the age far enough (breaker.F:182-224)
template <typename T>
__device__ __forceinline__ bool brk_try(const Grid &g, const Fields<T> &f, volatile T *N, int code, T DT) {
    const int i = code % g.pitch, j = code / g.pitch;
    const size_t id = IDX(i, j);
    if (N[id] != (T)0 || !brk_neigh(g, f, N, i, j, DT)) return false;
    N[id] = DT;
    return true;
}

// exclusive prefix sum over a 1024-thread block (wsum: 32 ints of shared
// memory); returns this thread's prefix
__device__ __forceinline__ int block_scan_1024(int x, int *wsum) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int inc = x;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += y;
    }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const int w = wsum[lane];
        int wi = w;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, wi, d);
            if (lane >= d) wi += y;
        }
        wsum[lane] = wi - w;
    }
    __syncthreads();
    const int r = wsum[warp] + inc - x;
    __syncthreads();
    return r;
}

// Candidates of the sweep, in one 1024-thread block, then nu.  The sweep
// (j outer, i inner) lets a candidate read the new values of (i-1,j),
// (i-1,j-1), (i,j-1), (i+1,j-1) (cells before it) and the old values of
// the cells after it, so new values only flow forward and a candidate
// turns from 0 to DT at most once.
//  - Passes to the fixed point: every candidate tests its neighbours in
//    parallel, and the pass repeats while any changed.  What a pass sets
//    is also set by the sequential sweep (by induction over the passes),
//    so the fixed point is its result.  A chain of k candidates that set
//    one another takes k + 1 passes; most stages need two or three.
//  - After g.brk_passes passes without the fixed point, the rest in one
//    pass by level t = i + 2j: the cells a candidate reads new values of
//    lie on levels t-1, t-3, t-2, t-1, the cells it reads old values of on
//    levels above t.  The candidates are sorted by level (a histogram, its
//    prefix sum and a scatter, into the line solver's tp plane, which is
//    free between the stage's line solve and the next) and the
//    non-empty levels are worked in order, one barrier each.  Starting
//    from any pass's state (a subset of the sweep's result) this gives the
//    sweep's result, in time bounded by the candidates and the levels
//    (at most Mglob + 2 Nglob + 7) whatever the breaking pattern.
template <typename T>
__global__ void __launch_bounds__(1024) k_break_b(Grid g, Fields<T> f) {
    __shared__ int changed;
    __shared__ int wsum[32];
    __shared__ int lev_beg[1024], lev_end[1024];
    __shared__ unsigned nonempty[32];
    const int n = (int)min((unsigned)*f.ncand, (unsigned)cand_cap(g));
    const T DT = DTV;
    volatile T *N = f.AGEn;
    bool done = false;
    for (int pass = 0; pass < g.brk_passes && pass <= n; pass++) {
        if (threadIdx.x == 0) changed = 0;
        __syncthreads();
        for (int c = threadIdx.x; c < n; c += blockDim.x)
            if (brk_try(g, f, N, f.cand[c], DT)) changed = 1;
        __syncthreads();
        const int ch = changed;
        __syncthreads();
        if (!ch) {
            done = true;
            break;
        }
    }
    if (!done && n > 0) {
        // levels of the candidate range Ibeg-1..Iend+1 x Jbeg-1..Jend+1
        const int i0 = g.ib - 1, j0 = g.jb - 1;
        const int nlev = (g.ie + 1 - i0) + 2 * (g.je + 1 - j0) + 1;
        // a plane of doubles holds two planes of ints
        int *sorted = reinterpret_cast<int *>(f.tp);
        int *off_a = sorted + (size_t)g.pitch * (size_t)(g.Nloc + 1);
        volatile int *off = off_a;
        auto level = [&](int code) { return (code % g.pitch - i0) + 2 * (code / g.pitch - j0); };
        for (int t = threadIdx.x; t < nlev; t += 1024) off[t] = 0;
        __syncthreads();
        for (int c = threadIdx.x; c < n; c += 1024) atomicAdd(&off_a[level(f.cand[c])], 1);
        __syncthreads();
        // counts -> exclusive offsets: each thread takes a run of levels
        const int per = (nlev + 1023) / 1024;
        const int lo = min((int)threadIdx.x * per, nlev), hi = min(lo + per, nlev);
        int sum = 0;
        for (int t = lo; t < hi; t++) sum += off[t];
        int acc = block_scan_1024(sum, wsum);
        for (int t = lo; t < hi; t++) {
            const int v = off[t];
            off[t] = acc;
            acc += v;
        }
        __syncthreads();
        // scatter; afterwards off[t] is the end of level t
        for (int c = threadIdx.x; c < n; c += 1024) {
            const int code = f.cand[c];
            sorted[atomicAdd(&off_a[level(code)], 1)] = code;
        }
        __syncthreads();
        // the levels in order, 1024 at a time: each thread flags its level
        // if non-empty, and all threads walk the same flags, so every
        // thread reaches the same barriers
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        for (int t0 = 0; t0 < nlev; t0 += 1024) {
            const int t = t0 + threadIdx.x;
            int b = 0, e = 0;
            if (t < nlev) {
                e = off[t];
                b = t == 0 ? 0 : off[t - 1];
            }
            lev_beg[threadIdx.x] = b;
            lev_end[threadIdx.x] = e;
            const unsigned m = __ballot_sync(0xffffffffu, e > b);
            if (lane == 0) nonempty[warp] = m;
            __syncthreads();
            for (int w = 0; w < 32; w++) {
                unsigned mw = nonempty[w];
                while (mw) {
                    const int k = w * 32 + __ffs(mw) - 1;
                    mw &= mw - 1;
                    for (int c = lev_beg[k] + threadIdx.x; c < lev_end[k]; c += 1024)
                        brk_try(g, f, N, sorted[c], DT);
                    __syncthreads();
                }
            }
            __syncthreads();  // all have read the flags before the next chunk's
        }
    }
    for (int c = threadIdx.x; c < n; c += blockDim.x) {
        const int code = f.cand[c];
        const int i = code % g.pitch, j = code / g.pitch;
        const size_t id = IDX(i, j);
        if (in_wk_zone<T>(g, i, j)) continue;
        const BrkLocal<T> b = brk_local(g, f, id);
        f.nu[id] = nu_value(g, f, id, b, (T)N[id], false);
        if (g.track_roller && breaking_now(g, b, (T)N[id])) roller_cell(g, f, id, b.et);
    }
    __syncthreads();
    if (threadIdx.x == 0) *f.ncand = 0;
}

// ---------------------------------------------------------------------------
// EXCHANGE ghost fill (bc.F:426-529 with PHI_COLL / PHI_COLL_VARIABLE_LENGTH)
// in place.  One thread per ghost cell; in periodic mode the thread of an
// x-ghost cell also moves its pre-fill value into the corner cell that
// copies it (bc.F:735-740 runs before the x mirror).
// ---------------------------------------------------------------------------
struct GhostSet {
    int n;  // number of fields
};

template <typename T>
__device__ __forceinline__ void ghost_x_cell(const Grid &g, T *phi, int i, int j, int vtype) {
    // i is an x-ghost column, j an interior row
    const int si = mirror_x(g, i);
    const T v = phi[IDX(si, j)];
    if (g.periodic) {
        if (j >= g.je - 2) phi[IDX(i, j - (g.je - 2))] = phi[IDX(i, j)];
        if (j <= g.jb + 2) phi[IDX(i, j + g.je - 2)] = phi[IDX(i, j)];
    }
    phi[IDX(i, j)] = (vtype == 2) ? -v : v;
}
template <typename T>
__device__ __forceinline__ void ghost_y_cell(const Grid &g, T *phi, int i, int j, int vtype) {
    // j is a y-ghost row, any column
    const bool gx = (i < g.ib) || (i > g.ie);
    if (g.periodic) {
        if (gx) return;  // corner: written by the x-ghost thread
        phi[IDX(i, j)] = phi[IDX(i, period_y(g, j))];
        return;
    }
    const T v = phi[IDX(mirror_x(g, i), mirror_y(g, j))];
    T r = v;
    if (vtype == 2 && gx) r = -r;
    if (vtype == 3) r = -r;
    phi[IDX(i, j)] = r;
}

// EXCHANGE's PHI_COLL of Wsurf, P_center, Q_center, U_davg and V_davg
// (bc.F:438-443), scalar rules, after the last two stages
template <typename T>
__global__ void __launch_bounds__(256) k_ghost_rad(Grid g, Fields<T> f) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int nX = 6 * g.Nglob, nY = 6 * g.Mloc;
    if (t >= nX + nY) return;
    const size_t PL = (size_t)g.pitch * (size_t)(g.Nloc + 1);
    T *const planes[5] = {f.rad + RP_WS * PL, f.rad + RP_PC * PL, f.rad + RP_QC * PL, f.rad + RP_UD * PL,
                          f.rad + RP_VD * PL};
    if (t < nX) {
        const int col = t % 6;
        const int i = col < 3 ? col : g.ie + 1 + (col - 3);
        const int j = g.jb + t / 6;
#pragma unroll
        for (int k = 0; k < 5; k++) ghost_x_cell(g, planes[k], i, j, 1);
    } else {
        const int u = t - nX;
        const int row = u / g.Mloc;
        const int i = u % g.Mloc;
        const int j = row < 3 ? row : g.je + 1 + (row - 3);
#pragma unroll
        for (int k = 0; k < 5; k++) ghost_y_cell(g, planes[k], i, j, 1);
    }
}

template <typename T>
__global__ void __launch_bounds__(256) k_ghost(Grid g, Fields<T> f, int with_age) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int nX = 6 * g.Nglob;
    const int nY = 6 * g.Mloc;
    const int ncell = nX + nY;
    if (t < ncell) {
        if (t < nX) {
            const int col = t % 6;
            const int i = col < 3 ? col : g.ie + 1 + (col - 3);
            const int j = g.jb + t / 6;
            ghost_x_cell(g, f.Eta, i, j, 1);
            ghost_x_cell(g, f.U, i, j, 2);
            ghost_x_cell(g, f.HU, i, j, 2);
            ghost_x_cell(g, f.V, i, j, 3);
            ghost_x_cell(g, f.HV, i, j, 3);
            ghost_x_cell(g, f.MASK, i, j, 1);
            if (with_age) {
                ghost_x_cell(g, f.AGE, i, j, 1);
                ghost_x_cell(g, f.nu, i, j, 1);
            }
        } else {
            const int u = t - nX;
            const int row = u / g.Mloc;
            const int i = u % g.Mloc;
            const int j = row < 3 ? row : g.je + 1 + (row - 3);
            ghost_y_cell(g, f.Eta, i, j, 1);
            ghost_y_cell(g, f.U, i, j, 2);
            ghost_y_cell(g, f.HU, i, j, 2);
            ghost_y_cell(g, f.V, i, j, 3);
            ghost_y_cell(g, f.HV, i, j, 3);
            ghost_y_cell(g, f.MASK, i, j, 1);
            if (with_age) {
                ghost_y_cell(g, f.AGE, i, j, 1);
                ghost_y_cell(g, f.nu, i, j, 1);
            }
        }
        return;
    }
    if (!with_age) return;
    // P on x-faces and Q on y-faces: plain mirror on all four sides
    // (PHI_COLL_VARIABLE_LENGTH, periodic ignored), last index Iend1 / Jend1
    int u = t - ncell;
    const int nPX = 6 * g.Nglob, nPY = 6 * (g.Mloc + 1);
    if (u < nPX + nPY) {
        const int ie1 = g.ie + 1;
        int i, j;
        if (u < nPX) {
            const int col = u % 6;
            i = col < 3 ? col : ie1 + 1 + (col - 3);
            j = g.jb + u / 6;
        } else {
            u -= nPX;
            const int row = u / (g.Mloc + 1);
            i = u % (g.Mloc + 1);
            j = row < 3 ? row : g.je + 1 + (row - 3);
        }
        const int si = i < g.ib ? 2 * g.ib - 1 - i : (i > ie1 ? 2 * ie1 + 1 - i : i);
        const int sj = mirror_y(g, j);
        f.P[IDX(i, j)] = f.P[IDX(si, sj)];
        return;
    }
    u -= nPX + nPY;
    const int nQX = 6 * (g.Nglob + 1), nQY = 6 * g.Mloc;
    if (u < nQX + nQY) {
        const int je1 = g.je + 1;
        int i, j;
        if (u < nQX) {
            const int col = u % 6;
            i = col < 3 ? col : g.ie + 1 + (col - 3);
            j = g.jb + u / 6;
        } else {
            u -= nQX;
            const int row = u / g.Mloc;
            i = u % g.Mloc;
            j = row < 3 ? row : je1 + 1 + (row - 3);
        }
        const int si = mirror_x(g, i);
        const int sj = j < g.jb ? 2 * g.jb - 1 - j : (j > je1 ? 2 * je1 + 1 - j : j);
        f.Q[IDX(i, j)] = f.Q[IDX(si, sj)];
    }
}

// U,V,HU,HV *= MASK (bc.F:491-494) and, optionally, SPONGE_DAMPING
// (sponge.F:52-66), on every cell
template <typename T>
__global__ void __launch_bounds__(256) k_maskmul(Grid g, Fields<T> f, int sponge) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= g.Mloc || j >= g.Nloc) return;
    const size_t id = IDX(i, j);
    // every load before the first store (see k_begin)
    const uint8_t mi = f.MASK[id];
    const T m = m2r<T>(mi);
    const T u0 = f.U[id], v0 = f.V[id], hu = f.HU[id], hv = f.HV[id];
    const T s = sponge ? f.SPONGE[id] : (T)1;
    const T eta = (sponge && mi > 0) ? f.Eta[id] : (T)0;
    T u = u0 * m, v = v0 * m;
    f.HU[id] = hu * m;
    f.HV[id] = hv * m;
    if (sponge) {
        if (mi > 0) f.Eta[id] = eta / s;
        u = u / s;
        v = v / s;
    }
    f.U[id] = u;
    f.V[id] = v;
}

// SPONGE_DAMPING alone
template <typename T>
__global__ void k_sponge(Grid g, Fields<T> f) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= g.Mloc || j >= g.Nloc) return;
    const size_t id = IDX(i, j);
    const T s = f.SPONGE[id];
    if (f.MASK[id] > 0) f.Eta[id] = f.Eta[id] / s;
    f.U[id] = f.U[id] / s;
    f.V[id] = f.V[id] / s;
}

// ---------------------------------------------------------------------------
// ESTIMATE_DT (misc.F:216-296): CFL minimum over every cell, then DT and
// TIME on the device.  Positive doubles order like their bit patterns.
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ T dt_val(const Grid &g, T H, T U, T V) {
    const T c = fsqrt((T)GRAV * tmax(H, GC(min_depth_frc)));
    T t1 = fabs_(U) + c;
    T t2 = (t1 < (T)SMALL) ? GC(DX) / (T)SMALL : GC(DX) / t1;
    T m = t2;
    t1 = fabs_(V) + c;
    t2 = (t1 < (T)SMALL) ? GC(DY) / (T)SMALL : GC(DY) / t1;
    if (t2 < m) m = t2;
    return m;
}
template <typename T>
__device__ __forceinline__ T dt_cell(const Grid &g, const Fields<T> &f, size_t id) {
    return dt_val(g, f.H[id], f.U[id], f.V[id]);
}

__device__ __forceinline__ double tminr(double a, double b) { return fmin(a, b); }
__device__ __forceinline__ float tminr(float a, float b) { return fminf(a, b); }

// block minimum in T, then one atomicMin on the (order-preserving) bits of
// the positive double
template <typename T>
__device__ __forceinline__ void block_min_to_global(T v, unsigned long long *dst) {
    __shared__ T sm[32];
    for (int o = 16; o > 0; o >>= 1) v = tminr(v, __shfl_xor_sync(0xffffffffu, v, o));
    const int lane = (threadIdx.x + threadIdx.y * blockDim.x) & 31;
    const int warp = (threadIdx.x + threadIdx.y * blockDim.x) >> 5;
    const int nw = (blockDim.x * blockDim.y + 31) >> 5;
    if (lane == 0) sm[warp] = v;
    __syncthreads();
    if (warp == 0) {
        v = lane < nw ? sm[lane] : (T)1.0e30;
        for (int o = 16; o > 0; o >>= 1) v = tminr(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane == 0) atomicMin(dst, (unsigned long long)__double_as_longlong((double)v));
    }
}

// Eta0 = Eta on the ghost ring, before the step's EXCHANGE refills it
// (main.F:295 comes before main.F:313): the ring still holds the previous
// step's sponge-damped values.  6*Mloc + 6*Nglob cells, one thread each.
template <typename T>
__global__ void __launch_bounds__(256) k_eta0_ring(Grid g, Fields<T> f) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    int i, j;
    if (t < 3 * g.Mloc) {
        j = t / g.Mloc;
        i = t - j * g.Mloc;
    } else if ((t -= 3 * g.Mloc) < 3 * g.Mloc) {
        j = g.Nloc - 3 + t / g.Mloc;
        i = t % g.Mloc;
    } else if ((t -= 3 * g.Mloc) < 6 * g.Nglob) {
        j = NG + t / 6;
        const int c = t % 6;
        i = c < 3 ? c : g.Mloc - 6 + c;
    } else {
        return;
    }
    f.Eta0[IDX(i, j)] = f.Eta[IDX(i, j)];
}

// begin of a step: U,V,HU,HV *= MASK after the ghost fill, the Eta0
// (interior; the ring is copied by k_eta0_ring before the fill), Ubar0,
// Vbar0, U0, V0 copies (main.F:295-297,331) and the CFL minimum
template <typename T>
__global__ void __launch_bounds__(256) k_begin(Grid g, Fields<T> f) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    T v = (T)1.0e30;
    if (i < g.Mloc && j < g.Nloc) {
        const size_t id = IDX(i, j);
        // every load before the first store: the copies' sources and
        // destinations are different arrays, which the compiler cannot know
        const bool in = i >= g.ib && i <= g.ie && j >= g.jb && j <= g.je;
        const T m = m2r<T>(f.MASK[id]);
        const T u0 = f.U[id], v0 = f.V[id], hu = f.HU[id], hv = f.HV[id];
        const T ub = f.Ubar[id], vb = f.Vbar[id], h = f.H[id];
        const T eta = in ? f.Eta[id] : (T)0;
        const T u = u0 * m, vv = v0 * m;
        f.U[id] = u;
        f.V[id] = vv;
        f.HU[id] = hu * m;
        f.HV[id] = hv * m;
        if (in) f.Eta0[id] = eta;
        f.Ubar0[id] = ub;
        f.Vbar0[id] = vb;
        f.U0[id] = u;
        f.V0[id] = vv;
        v = dt_val(g, h, u, vv);
    }
    block_min_to_global(v, f.dtmin_bits);
}

// EXCHANGE in one pass, for grids of at least 3 x 3: the ghost fill (k_ghost),
// then U,V,HU,HV *= MASK and SPONGE_DAMPING (k_maskmul), or at the begin of a
// step k_eta0_ring, the fill and k_begin.  The thread of an interior cell
// writes its own cell and the ghost cells that take their values from it (at
// most three along each axis and their corner), so that no thread reads what
// another writes.  With PERIODIC the ghost corners take the x ghost's value
// from before its fill (bc.F:735-740), which the same thread reads first.
// The rows of blocks before the last nby fill P's and Q's ghosts
// (PHI_COLL_VARIABLE_LENGTH).
// The fill as a launch of its own took 7-10 us (a chain of eight loads and
// stores on a few thousand threads), four times a step: 20 steps of 250 x 500
// 4181 -> 3879 us.
template <typename T> struct ExCell {
    T eta, u, v, hu, hv, age, nu;
    uint8_t m;
};
template <typename T> __device__ __forceinline__ void ghost_pq(const Grid &g, const Fields<T> &f, int u) {
    const int nPX = 6 * g.Nglob, nPY = 6 * (g.Mloc + 1);
    int i, j;
    if (u < nPX + nPY) {
        const int ie1 = g.ie + 1;
        if (u < nPX) {
            const int col = u % 6;
            i = col < 3 ? col : ie1 + 1 + (col - 3);
            j = g.jb + u / 6;
        } else {
            u -= nPX;
            const int row = u / (g.Mloc + 1);
            i = u % (g.Mloc + 1);
            j = row < 3 ? row : g.je + 1 + (row - 3);
        }
        const int si = i < g.ib ? 2 * g.ib - 1 - i : (i > ie1 ? 2 * ie1 + 1 - i : i);
        f.P[IDX(i, j)] = f.P[IDX(si, mirror_y(g, j))];
        return;
    }
    u -= nPX + nPY;
    const int nQX = 6 * (g.Nglob + 1), nQY = 6 * g.Mloc;
    if (u < nQX + nQY) {
        const int je1 = g.je + 1;
        if (u < nQX) {
            const int col = u % 6;
            i = col < 3 ? col : g.ie + 1 + (col - 3);
            j = g.jb + u / 6;
        } else {
            u -= nQX;
            const int row = u / g.Mloc;
            i = u % g.Mloc;
            j = row < 3 ? row : je1 + 1 + (row - 3);
        }
        const int sj = j < g.jb ? 2 * g.jb - 1 - j : (j > je1 ? 2 * je1 + 1 - j : j);
        f.Q[IDX(i, j)] = f.Q[IDX(mirror_x(g, i), sj)];
    }
}
// one cell as the fill leaves it, masked and damped; own: the interior cell
// itself (its MASK, AGE and nu stay).  Returns the cell's CFL value (BEGIN).
template <typename T, bool BEGIN>
__device__ __forceinline__ T ex_put(const Grid &g, const Fields<T> &f, int id, const ExCell<T> &c, bool own, int sponge,
                                    int with_age) {
    // every load before the first use of a loaded value
    T h = (T)0, ub = (T)0, vb = (T)0, e0 = c.eta, s = (T)1;
    if (BEGIN) {
        h = f.H[id];
        ub = f.Ubar[id];
        vb = f.Vbar[id];
        if (!own) e0 = f.Eta[id];
    } else if (sponge) {
        s = f.SPONGE[id];
    }
    const T m = m2r<T>(c.m);
    T u = c.u * m, v = c.v * m, eta = c.eta, r = (T)1.0e30;
    if (BEGIN) {
        f.Eta0[id] = e0;
        f.Ubar0[id] = ub;
        f.Vbar0[id] = vb;
        f.U0[id] = u;
        f.V0[id] = v;
        r = dt_val(g, h, u, v);
    } else if (s != (T)1) {  // 1 outside the sponges: nothing to divide
        if (c.m > 0) eta = eta / s;
        u = u / s;
        v = v / s;
    }
    f.U[id] = u;
    f.V[id] = v;
    f.HU[id] = c.hu * m;
    f.HV[id] = c.hv * m;
    if (!own || (!BEGIN && sponge)) f.Eta[id] = eta;
    if (!own) {
        f.MASK[id] = c.m;
        if (with_age) {
            f.AGE[id] = c.age;
            f.nu[id] = c.nu;
        }
    }
    return r;
}
// (seven blocks to an SM, 36 registers: 41 -> 35 us at 2048 x 2048; the begin's
// twelve streams want the registers: 62 us, 68 with seven)
template <typename T, bool BEGIN>
__global__ void __launch_bounds__(256, !BEGIN && sizeof(T) == sizeof(float) ? 7 : 1) k_exchange(Grid g, Fields<T> f, int sponge, int with_age, int nby, Ahead ah) {
    const int npq = (int)gridDim.y - nby;
    int by = (int)blockIdx.y - npq;
    if (by < 0) {
        const int nt = blockDim.x * blockDim.y;
        ghost_pq(g, f, ((int)blockIdx.y * (int)gridDim.x + (int)blockIdx.x) * nt + threadIdx.x + threadIdx.y * blockDim.x);
        return;
    }
    // the rows with ghost images, which take longest, first: 0, last, 1, 2, ..
    if (by >= 2) prefetch_ahead<T>(g, ah, by - 1, g.jb);
    if (by > 0) by = by == 1 ? nby - 1 : by - 1;
    // columns from 0: whole 128-byte lines to a warp
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = g.jb + by * blockDim.y + threadIdx.y;
    T dt = (T)1.0e30;
    if (i >= g.ib && i <= g.ie && j <= g.je) {
        const int id = i + j * g.pitch;
        ExCell<T> c;
        c.m = f.MASK[id];
        c.u = f.U[id];
        c.v = f.V[id];
        c.hu = f.HU[id];
        c.hv = f.HV[id];
        c.eta = f.Eta[id];
        c.age = c.nu = (T)0;
        const bool xl = i < g.ib + 3, xr = i > g.ie - 3, yl = j < g.jb + 3, yr = j > g.je - 3;
        const bool edge = xl || xr || yl || yr;
        if (edge && with_age) {
            c.age = f.AGE[id];
            c.nu = f.nu[id];
        }
        dt = ex_put<T, BEGIN>(g, f, id, c, true, sponge, with_age);
        if (edge) {
            // the ghost rows and columns that take their values from this cell
            const int gx[2] = {xl ? 2 * g.ib - 1 - i : -1, xr ? 2 * g.ie + 1 - i : -1};
            const int gy[2] = {yl ? (g.periodic ? j + g.je - 2 : 2 * g.jb - 1 - j) : -1,
                               yr ? (g.periodic ? j - (g.je - 2) : 2 * g.je + 1 - j) : -1};
            const T sy = g.periodic ? (T)1 : (T)-1;
            auto signs = [&](T su, T sv) {
                ExCell<T> d = c;
                d.u = su * c.u;
                d.hu = su * c.hu;
                d.v = sv * c.v;
                d.hv = sv * c.hv;
                return d;
            };
#pragma unroll
            for (int a = 0; a < 2; a++) {
                if (gx[a] < 0) continue;
                const int gid = gx[a] + j * g.pitch;
                if (g.periodic && (yl || yr)) {
                    ExCell<T> o;
                    o.m = f.MASK[gid];
                    o.u = f.U[gid];
                    o.v = f.V[gid];
                    o.hu = f.HU[gid];
                    o.hv = f.HV[gid];
                    o.eta = f.Eta[gid];
                    o.age = with_age ? f.AGE[gid] : (T)0;
                    o.nu = with_age ? f.nu[gid] : (T)0;
#pragma unroll
                    for (int b = 0; b < 2; b++)
                        if (gy[b] >= 0)
                            dt = tminr(dt, ex_put<T, BEGIN>(g, f, gx[a] + gy[b] * g.pitch, o, false, sponge, with_age));
                }
                dt = tminr(dt, ex_put<T, BEGIN>(g, f, gid, signs((T)-1, (T)1), false, sponge, with_age));
                if (!g.periodic) {
#pragma unroll
                    for (int b = 0; b < 2; b++)
                        if (gy[b] >= 0)
                            dt = tminr(dt, ex_put<T, BEGIN>(g, f, gx[a] + gy[b] * g.pitch, signs((T)-1, sy), false, sponge,
                                                           with_age));
                }
            }
#pragma unroll
            for (int b = 0; b < 2; b++)
                if (gy[b] >= 0)
                    dt = tminr(dt, ex_put<T, BEGIN>(g, f, i + gy[b] * g.pitch, signs((T)1, sy), false, sponge, with_age));
        }
    }
    if (BEGIN) block_min_to_global(dt, f.dtmin_bits);
}

template <typename T>
__global__ void __launch_bounds__(256) k_dt_only(Grid g, Fields<T> f) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    T v = (T)1.0e30;
    if (i < g.Mloc && j < g.Nloc) v = dt_cell(g, f, IDX(i, j));
    block_min_to_global(v, f.dtmin_bits);
}

// DT = CFL*min (with DT_fixed halving), TIME += DT, and the JON_2D
// cos/sin(omega_k TIME) table of this step (sources.F:121-124)
static __global__ void k_dt_final(Grid g, double *dsc, float *fsc, unsigned long long *bits, double *omega,
                                  double *wmcs, float *wmcsf, int nfreq) {
    __shared__ double time_s;
    if (threadIdx.x == 0) {
        double tmp3 = __longlong_as_double((long long)*bits);
        if (!(tmp3 < LARGE)) tmp3 = LARGE;
        const double dt_tmp = g.cfl * tmp3;
        double dt;
        if (g.fixed_dt) {
            dt = g.dt_fixed;
            for (int k = 0; k < 4096 && dt > dt_tmp; k++) dt = dt / 2.0;
        } else {
            dt = dt_tmp;
        }
        dsc[S_DT] = dt;
        dsc[S_TIME] = dsc[S_TIME] + dt;
        time_s = dsc[S_TIME];
        *bits = 0x7ff0000000000000ull;  // +inf for the next minimum
        // float scalars of the step for the mixed path: DT, 1/DT, the
        // wavemaker ramp (sources.F:110,120) and the WK_REG phase
        // 2*pi/Tperiod*TIME reduced modulo 2*pi
        fsc[FS_DT] = (float)dt;
        fsc[FS_RDT] = (float)(1.0 / dt);
        if (g.wavemaker == FW_WK_REG) {
            fsc[FS_WKAA] = (float)(tanh(PI_SP / (g.time_ramp * g.tperiod) * time_s) * g.D_gen);
            const double ph = 2.0 * PI_SP / g.tperiod * time_s;
            fsc[FS_WKPH] = (float)(ph - 2.0 * PI_SP * floor(ph / (2.0 * PI_SP)));
        } else if (g.wavemaker == FW_WK_JON_2D) {
            fsc[FS_WKAA] = (float)tanh(PI_SP / (g.time_ramp / g.freq_peak) * time_s);
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < nfreq; k += blockDim.x) {
        wmcs[2 * k] = cos(omega[k] * time_s);
        wmcs[2 * k + 1] = sin(omega[k] * time_s);
        wmcsf[2 * k] = (float)wmcs[2 * k];
        wmcsf[2 * k + 1] = (float)wmcs[2 * k + 1];
    }
}

// ---------------------------------------------------------------------------
// end of a step: MAX_MIN_PROPERTY (Hmax, misc.F:307-383) and the
// CHECK_BLOWUP maximum (misc.F:394-433)
// ---------------------------------------------------------------------------
// MIXING_STUFF's T_sum (mixing.F:60, 143-144, 224): one thread, before
// k_end; S_MFLAG tells k_end what to do with the cells this step
static __global__ void k_tsum(Grid g, double *dsc, float *fsc) {
    int flag = 0;
    double ts = dsc[S_TSUM], tsu = ts;
    if (dsc[S_TIME] >= g.steady_time) {
        ts = ts + dsc[S_DT];
        tsu = ts;
        if (ts >= g.t_intv_mean) {
            flag = 2;
            ts = ts - g.t_intv_mean;
            dsc[S_NMEAN] = dsc[S_NMEAN] + 1.0;
        } else {
            flag = 1;
        }
    }
    dsc[S_TSUM] = ts;
    dsc[S_TSUMU] = tsu;
    dsc[S_MFLAG] = (double)flag;
    fsc[FS_TSUM] = (float)tsu;
}

// s += x with Kahan compensation k (mixed path), s = x + s otherwise
template <typename T> __device__ __forceinline__ void stat_add(T *s, T *k, size_t id, T x) {
    if constexpr (sizeof(T) == sizeof(double)) {
        s[id] = x + s[id];
    } else {
        const float y = __fsub_rn(x, k[id]);
        const float t = __fadd_rn(s[id], y);
        k[id] = __fsub_rn(__fsub_rn(t, s[id]), y);
        s[id] = t;
    }
}
// the compensated value of a sum
template <typename T> __device__ __forceinline__ T stat_val(const T *s, const T *k, size_t id) {
    if constexpr (sizeof(T) == sizeof(double)) return s[id];
    else return __fsub_rn(s[id], k[id]);
}

// CALCULATE_MEAN's radiation-stress, momentum-flux and breaking-dissipation
// sums at one cell (mixing.F:156-167, 270-281), with the ETAmean the
// caller's branch has at that point and the last interval's U_davg_mean
template <typename T> __device__ __forceinline__ void rad_sums(const Grid &g, const Fields<T> &f, size_t id, T DT,
                                                               T etamean) {
    const size_t PL = (size_t)g.pitch * (size_t)(g.Nloc + 1);
    T *const r = f.rad;
    T *const ks = sizeof(T) == sizeof(float) ? r + RP_KAHAN * PL : nullptr;
#define RV(k) r[(size_t)(k) * PL + id]
#define SUM(k, x) stat_add(r + (RP_SUM + (k)) * PL, ks ? ks + (size_t)(k) * PL : nullptr, id, (T)(x))
    const T udv = RV(RP_UD), vdv = RV(RP_VD);
    const T ud = udv - RV(RP_MEAN + 0), vd = vdv - RV(RP_MEAN + 1);
    const T hd = f.Eta[id] - etamean + f.Depth[id];
    const T u = f.U[id], v = f.V[id], w = RV(RP_WS);
    const T sp = fsqrt(u * u + v * v);
    SUM(0, udv * DT);
    SUM(1, vdv * DT);
    SUM(2, RV(RP_PC) * DT);
    SUM(3, RV(RP_QC) * DT);
    SUM(4, ud * ud * hd * DT);
    SUM(5, ud * vd * hd * DT);
    SUM(6, vd * vd * hd * DT);
    SUM(7, (T)0.25 * w * w * hd * DT);
    SUM(8, u * sp * DT);
    SUM(9, v * sp * DT);
    SUM(10, RV(RP_BX) * DT);
    SUM(11, RV(RP_BY) * DT);
#undef SUM
#undef RV
}
// the means at the end of an interval, then the sums restart
template <typename T> __device__ __forceinline__ void rad_means(const Grid &g, const Fields<T> &f, size_t id, T Ts) {
    const size_t PL = (size_t)g.pitch * (size_t)(g.Nloc + 1);
    T *const r = f.rad;
#pragma unroll
    for (int k = 0; k < 12; k++) {
        T *s = r + (RP_SUM + k) * PL;
        T *kk = sizeof(T) == sizeof(float) ? r + (RP_KAHAN + k) * PL : nullptr;
        r[(RP_MEAN + k) * PL + id] = stat_val(s, kk, id) / Ts;
        s[id] = (T)0;
        if (kk) kk[id] = (T)0;
    }
}

// CALCULATE_MEAN (mixing.F:141-301) at one cell: the Eta, U, V and
// (Eta-ETAmean)^2 time sums, their means at the end of an interval, and the
// zero-up-crossing wave heights; the float path keeps the sums compensated
template <typename T> __device__ __forceinline__ void mean_cell(const Grid &g, const Fields<T> &f, size_t id,
                                                                int flag) {
    const T DT = DTV;
    // Each sum is read, added to and stored behind the one before it; their
    // lines are asked for together first (997 x 1501 with the radiation sums:
    // k_end 122 -> 101 us.  Loading them all into registers takes 175 of them
    // and 214 us, at 128 registers 168).
    constexpr bool KAHAN = sizeof(T) == sizeof(float);
    if (f.rad) {
        const size_t PL = (size_t)g.pitch * (size_t)(g.Nloc + 1);
        const T *r = f.rad + id;
#pragma unroll
        for (int k = 0; k < 12; k++) {
            prefetch_l1(r + (RP_SUM + k) * PL);
            if (KAHAN) prefetch_l1(r + (RP_KAHAN + k) * PL);
        }
        const int in[9] = {RP_UD, RP_VD, RP_PC, RP_QC, RP_WS, RP_BX, RP_BY, RP_MEAN, RP_MEAN + 1};
#pragma unroll
        for (int k = 0; k < 9; k++) prefetch_l1(r + in[k] * PL);
        prefetch_l1(f.Depth + id);
    }
    const T *const sums[7] = {f.Usum, f.Vsum, f.ETAsum, f.ETA2sum, f.Emax, f.Emin, f.Eta0};
#pragma unroll
    for (int k = 0; k < 7; k++) prefetch_l1(sums[k] + id);
    if (KAHAN) {
        const T *const ks[4] = {f.kUsum, f.kVsum, f.kETAsum, f.kETA2sum};
#pragma unroll
        for (int k = 0; k < 4; k++) prefetch_l1(ks[k] + id);
    }
    const T eta = f.Eta[id], u = f.U[id], v = f.V[id];
    const T d = eta - f.ETAmean[id];
    if (flag == 2) {
        T Ts;
        if constexpr (sizeof(T) == sizeof(double)) Ts = f.dsc[S_TSUMU];
        else Ts = f.fsc[FS_TSUM];
        stat_add(f.ETA2sum, f.kETA2sum, id, d * d * DT);
        const T e2 = stat_val(f.ETA2sum, f.kETA2sum, id) / Ts;
        f.ETA2mean[id] = e2;
        stat_add(f.Usum, f.kUsum, id, u * DT);
        stat_add(f.Vsum, f.kVsum, id, v * DT);
        stat_add(f.ETAsum, f.kETAsum, id, eta * DT);
        f.Umean[id] = stat_val(f.Usum, f.kUsum, id) / Ts;
        f.Vmean[id] = stat_val(f.Vsum, f.kVsum, id) / Ts;
        const T em = stat_val(f.ETAsum, f.kETAsum, id) / Ts;
        f.ETAmean[id] = em;
        if (f.rad) {
            rad_sums(g, f, id, DT, em);
            rad_means(g, f, id, Ts);
        }
        f.Usum[id] = (T)0;
        f.Vsum[id] = (T)0;
        f.ETAsum[id] = (T)0;
        f.ETA2sum[id] = (T)0;
        if constexpr (sizeof(T) == sizeof(float)) {
            f.kUsum[id] = 0.0f;
            f.kVsum[id] = 0.0f;
            f.kETAsum[id] = 0.0f;
            f.kETA2sum[id] = 0.0f;
        }
        f.SigWH[id] = (T)C4004_SP * fsqrt(e2);
        const T nz = f.NZU[id];
        if (nz >= (T)2) {
            f.WHave[id] = f.HavgSum[id] / nz;
            f.WHrms[id] = fsqrt(f.HrmsSum[id] / nz);
        }
    } else {
        stat_add(f.Usum, f.kUsum, id, u * DT);
        stat_add(f.Vsum, f.kVsum, id, v * DT);
        stat_add(f.ETAsum, f.kETAsum, id, eta * DT);
        stat_add(f.ETA2sum, f.kETA2sum, id, d * d * DT);
        if (f.rad) rad_sums(g, f, id, DT, f.ETAmean[id]);
        T emax = f.Emax[id], emin = f.Emin[id];
        if (eta > emax) emax = eta;
        if (eta < emin) emin = eta;
        const T tmp0 = f.Eta0[id] - f.ETAmean[id];
        if (d > tmp0 && d * tmp0 <= (T)0) {
            const T nz = f.NZU[id] + (T)1;
            f.NZU[id] = nz;
            if (nz >= (T)2) {
                const T h = emax - emin;
                f.HavgSum[id] = (f.HavgSum[id] + emax) - emin;  // left to right (mixing.F:293)
                f.HrmsSum[id] = f.HrmsSum[id] + h * h;
            }
            emax = (T)-1000;
            emin = (T)1000;
        }
        f.Emax[id] = emax;
        f.Emin[id] = emin;
    }
}

// the end of a CALCULATE_MEAN interval (mixing.F:183-219): the gradient
// fields DxSxx .. DxUVH of the new means on the interior, and FRCXmean,
// FRCYmean times Cd there.  Runs after k_end; a no-op on other steps.  The
// literals 9.80 and 0.5*9.80 are default REAL.
template <typename T>
__global__ void __launch_bounds__(256) k_rad_derived(Grid g, Fields<T> f) {
    if ((int)f.dsc[S_MFLAG] != 2) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x + g.ib;
    const int j = blockIdx.y * blockDim.y + threadIdx.y + g.jb;
    if (i > g.ie || j > g.je) return;
    const size_t PL = (size_t)g.pitch * (size_t)(g.Nloc + 1);
    const size_t id = IDX(i, j), e = IDX(i + 1, j), w = IDX(i - 1, j), n = IDX(i, j + 1), s = IDX(i, j - 1);
    T *const r = f.rad;
    const T *M = r + RP_MEAN * PL;
#define MN(k, c) M[(size_t)(k) * PL + (c)]
    const T DX = GC(DX), DY = GC(DY), mdf = GC(min_depth_frc);
    const T g98 = (T)9.80f, g49 = (T)(0.5f * 9.80f);
    const T *E2 = f.ETA2mean, *EM = f.ETAmean, *D = f.Depth;
    T *O = r + RP_DER * PL;
    // UU 4, UV 5, VV 6, WW 7; P 2, Q 3
    O[0 * PL + id] = (MN(4, e) - MN(4, w)) / (T)2 / DX - (MN(7, e) - MN(7, w)) / (T)2 / DX +
                     g49 * (E2[e] - E2[w]) / (T)2 / DX;
    O[1 * PL + id] = (MN(5, n) - MN(5, s)) / (T)2 / DY;
    O[2 * PL + id] = (MN(6, n) - MN(6, s)) / (T)2 / DY - (MN(7, n) - MN(7, s)) / (T)2 / DY +
                     g49 * (E2[n] - E2[s]) / (T)2 / DY;
    O[3 * PL + id] = (MN(5, e) - MN(5, w)) / (T)2 / DX;
    O[4 * PL + id] = g98 * (D[id] + EM[id]) * (EM[e] - EM[w]) / (T)2 / DX;
    O[5 * PL + id] = g98 * (D[id] + EM[id]) * (EM[n] - EM[s]) / (T)2 / DY;
    const T he = tmax(D[e] + EM[e], mdf), hw = tmax(D[w] + EM[w], mdf);
    const T hn = tmax(D[n] + EM[n], mdf), hs = tmax(D[s] + EM[s], mdf);
    O[6 * PL + id] = (MN(2, e) * MN(2, e) / he - MN(2, w) * MN(2, w) / hw) / (T)2 / DX;
    O[7 * PL + id] = (MN(2, n) * MN(3, n) / hn - MN(2, s) * MN(3, s) / hs) / (T)2 / DY;
    O[8 * PL + id] = (MN(3, n) * MN(3, n) / hn - MN(3, s) * MN(3, s) / hs) / (T)2 / DY;
    O[9 * PL + id] = (MN(2, e) * MN(3, e) / he - MN(2, w) * MN(3, w) / hw) / (T)2 / DX;
    T *FX = r + (RP_MEAN + 8) * PL, *FY = r + (RP_MEAN + 9) * PL;
    FX[id] = FX[id] * f.Cd[id];
    FY[id] = FY[id] * f.Cd[id];
#undef MN
}

template <typename T>
__global__ void __launch_bounds__(256) k_end(Grid g, Fields<T> f, int track_hmax) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    T v = (T)0;
    const int mflag = g.stats ? (int)f.dsc[S_MFLAG] : 0;
    if (i < g.Mloc && j < g.Nloc) {
        const size_t id = IDX(i, j);
        if (mflag) mean_cell(g, f, id, mflag);
        const T eta = f.Eta[id];
        // MAX_MIN_PROPERTY (misc.F:323-350), wet cells
        if (f.MASK[id] > 0) {
            if (track_hmax && eta > f.Hmax[id]) f.Hmax[id] = eta;
            if (g.track_hmin && eta < f.Hmin[id]) f.Hmin[id] = eta;
            if (g.track_umax || g.track_mfmax) {
                const T u = f.U[id], w = f.V[id];
                if (g.track_umax) {
                    const T mv = fsqrt(u * u + w * w);
                    if (mv > f.Umax[id]) f.Umax[id] = mv;
                }
                if (g.track_mfmax) {
                    const T mv = (u * u + w * w) * (f.H[id]);
                    if (mv > f.MFmax[id]) f.MFmax[id] = mv;
                }
            }
        }
        if (i >= g.ib && i <= g.ie && j >= g.jb && j <= g.je) {
            const T a = fabs_(eta);
            v = (a == a) ? a : (T)INFINITY;  // NaN -> +inf
        }
    }
    // block maximum, then one atomicMax per block on the (order-preserving)
    // bits of the non-negative double
    __shared__ T sm[32];
    for (int o = 16; o > 0; o >>= 1) {
        const T w = __shfl_xor_sync(0xffffffffu, v, o);
        v = w > v ? w : v;
    }
    const int t = threadIdx.x + threadIdx.y * blockDim.x;
    const int nw = (blockDim.x * blockDim.y + 31) >> 5;
    if ((t & 31) == 0) sm[t >> 5] = v;
    __syncthreads();
    if (t < 32) {
        v = t < nw ? sm[t] : (T)0;
        for (int o = 16; o > 0; o >>= 1) {
            const T w = __shfl_xor_sync(0xffffffffu, v, o);
            v = w > v ? w : v;
        }
        if (t == 0) atomicMax(f.etamax_bits, (unsigned long long)__double_as_longlong((double)v));
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
constexpr int GRID_Y_MAX = 65535;  // blocks of a launch along y
static inline dim3 grid2(int nx, int ny, dim3 b) { return dim3((nx + b.x - 1) / b.x, (ny + b.y - 1) / b.y); }
static const dim3 B2D(32, 8);
// blocks of k_flux_tma: tiles of FX x FY faces over (Mglob+1) x Nglob x-faces
// or Mglob x (Nglob+1) y-faces
template <typename T, int DIR, int FY_ = flux_fy_default<T, DIR>()> static dim3 flux_grid(const Grid &g) {
    using TL = FluxTile<T, DIR, FY_>;
    const int w = DIR == 0 ? g.Mglob + 1 : g.Mglob, h = DIR == 0 ? g.Nglob : g.Nglob + 1;
    return dim3((w + TL::FX - 1) / TL::FX, (h + TL::FY - 1) / TL::FY);
}

static inline void note(fw_ctx *c, int n = 1) {
    c->launches += n;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess && !c->sticky_error) c->sticky_error = (int)e;
}

// A captured step's launches that do not depend on one another go on two
// branches of its graph: the time step's end beside the first dispersion
// kernel, the factorisation (an early exit while MASK9 stands) beside the
// dispersion and the fluxes, the x fluxes beside the y fluxes and the x solve
// beside the y solve (they read the same planes and write their own).  On a
// small grid each of them leaves most of the GPU idle, on a large one the
// second fills the first one's last wave (a step of 128 x 256 cells 174 -> 143
// us, 250 x 500 194 -> 152, 2048 x 2048 2134 -> 2081; 250 x 500 in double 3186
// -> 3063, 701 x 937 11.0 -> 10.8 ms).
// Everything else stays on the context's stream, in the order of the step: a
// step outside a capture, and the entry points of single parts, any of which
// a caller may capture alone; such a capture must end with nothing on another
// stream and wait for nothing from outside it.
static bool branching(fw_ctx *c) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    return c->whole_step && !c->one_branch && cudaStreamIsCapturing(c->stream, &st) == cudaSuccess &&
           st == cudaStreamCaptureStatusActive;
}
// what `to` runs from here on comes after what `from` has so far
static void branch_after(fw_ctx *c, cudaStream_t to, cudaStream_t from, cudaEvent_t ev) {
    cudaError_t e = cudaEventRecord(ev, from);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(to, ev, 0);
    if (e != cudaSuccess && !c->sticky_error) c->sticky_error = (int)e;
}
// the launches of f on the side branch (behind what the step has so far), or
// in line
template <typename F> static void on_side(fw_ctx *c, bool branch, F f) {
    if (!branch) return f();
    cudaStream_t main = c->stream;
    branch_after(c, c->side, main, c->fork_ev);
    c->stream = c->side;
    f();
    c->stream = main;
}
static void join_side(fw_ctx *c, bool branch) {
    if (branch) branch_after(c, c->stream, c->side, c->join_ev);
}

template <typename T> void launch_ghost(fw_ctx *c, bool full) {
    const Grid &g = c->g;
    int n = 6 * g.Nglob + 6 * g.Mloc;
    if (full) n += 6 * g.Nglob + 6 * (g.Mloc + 1) + 6 * (g.Nglob + 1) + 6 * g.Mloc;
    k_ghost<T><<<(n + 255) / 256, 256, 0, c->stream>>>(g, c->F<T>(), full ? 1 : 0);
    note(c);
}

// Grids from which on a kernel brings lines ahead: where its inputs no longer
// come from the L2 anyway.  k_update, of 28 planes: 1024 x 1024 51.5 us with
// and 51.3 without, 1000 x 1500 60.7 and 64.3.  k_disp_a and
// k_post_mask_break: 1000 x 1500 24.7 and 24.5, 22.7 and 20.6; 1448 x 1448
// 36.9 and 39.3, 35.0 and 35.1.  k_exchange: 1448 x 1448 14.5 and 12.4; 2048 x
// 1500 20.7 and 20.5; 2048 x 2048 34.2 and 35.0.
constexpr long long AHEAD_UPDATE = 1LL << 20, AHEAD_A_PMB = 2LL << 20, AHEAD_EXCHANGE = 3LL << 20;
template <typename T> static void launch_disp_a(fw_ctx *c) {
    const Grid &g = c->g;
    const Fields<T> &f = c->F<T>();
    const dim3 b = c->blk(TK_DISP_A);
    const dim3 gr = grid2(g.Mloc, g.Nloc, b);
    k_disp_a<T><<<gr, b, 0, c->stream>>>(
        g, f, ahead_of<T>(g, b, gr.x, AHEAD_A_PMB, 2 * 152, {f.U, f.V, f.Depth, f.Eta, f.P, f.Q}));
}
// whether whole steps leave the wavemaker's mass to k_wm_band, and whether the
// launches under way are of one
template <typename T> static bool wm_has_band(fw_ctx *c) {
    return c->g.wavemaker == FW_WK_JON_2D && c->F<T>().Cm != nullptr;
}
template <typename T> static bool wm_in_band(fw_ctx *c) { return c->whole_step && wm_has_band<T>(c); }
template <typename T, bool RAD> static void launch_update(fw_ctx *c, T al, T be, bool band) {
    const Grid &g = c->g;
    const Fields<T> &f = c->F<T>();
    const dim3 b = c->blk(TK_UPDATE);
    const dim3 gr = grid2(g.Mloc, g.Nloc, b);
    auto kern = band ? k_update<T, RAD, true> : k_update<T, RAD, false>;
    kern<<<gr, b, 0, c->stream>>>(
        g, f, al, be,
        ahead_of<T>(g, b, gr.x, AHEAD_UPDATE, 2 * 152, {f.Eta0, f.Ubar0, f.Vbar0, f.Eta, f.Ubar, f.Vbar, f.P, f.Q, f.Fx, f.Fy, f.Gx, f.Gy,
                                              f.Depth, f.H, f.U, f.V, f.U4, f.V4, f.Depthx, f.Depthy, f.Udisp, f.Vdisp, f.U1p,
                                              f.V1p, f.Cd, f.HU, f.HV, f.nu}));
}
template <typename T> static void launch_pmb(fw_ctx *c) {
    const Grid &g = c->g;
    const Fields<T> &f = c->F<T>();
    const dim3 b = c->blk(TK_PMB);
    const dim3 gr = grid2(g.Mloc + 1, g.Nloc + 1, b);
    k_post_mask_break<T><<<gr, b, 0, c->stream>>>(
        g, f, ahead_of<T>(g, b, gr.x, AHEAD_A_PMB, 2 * 152, {f.U, f.V, f.H, f.AGE, f.Eta, f.Depth, f.ETAT}));
}

// EXCHANGE in one launch; false for grids too small for it, and for those
// whose rows of blocks and P's and Q's on top of them pass the launch limit
template <typename T, bool BEGIN> static bool launch_exchange_one(fw_ctx *c, bool sponge, dim3 b) {
    const Grid &g = c->g;
    if (g.Mglob < 3 || g.Nglob < 3) return false;
    const bool age = g.visc_breaking != 0;
    dim3 gr = grid2(g.ie + 1, g.Nglob, b);
    const int nby = (int)gr.y;
    if (age) {  // blocks for P's and Q's ghosts
        const int n = 6 * g.Nglob + 6 * (g.Mloc + 1) + 6 * (g.Nglob + 1) + 6 * g.Mloc, per = (int)(b.x * b.y * gr.x);
        gr.y += (n + per - 1) / per;
    }
    if (gr.y > GRID_Y_MAX) return false;
    const Fields<T> &f = c->F<T>();
    const Ahead ah = BEGIN ? ahead_of<T>(g, b, gr.x, AHEAD_EXCHANGE, 4 * 152, {f.U, f.V, f.HU, f.HV, f.Eta, f.H, f.Ubar, f.Vbar})
                           : ahead_of<T>(g, b, gr.x, AHEAD_EXCHANGE, 4 * 152, {f.U, f.V, f.HU, f.HV, f.Eta});
    k_exchange<T, BEGIN><<<gr, b, 0, c->stream>>>(g, f, sponge ? 1 : 0, age ? 1 : 0, nby, ah);
    note(c);
    return true;
}

template <typename T> void launch_exchange(fw_ctx *c, bool with_sponge) {
    const Grid &g = c->g;
    if (launch_exchange_one<T, false>(c, with_sponge, c->blk(TK_MASKMUL))) return;
    launch_ghost<T>(c, g.visc_breaking != 0);
    k_maskmul<T><<<grid2(g.Mloc, g.Nloc, c->blk(TK_MASKMUL)), c->blk(TK_MASKMUL), 0, c->stream>>>(g, c->F<T>(), with_sponge ? 1 : 0);
    note(c);
}

template <typename T> void launch_sponge(fw_ctx *c) {
    const Grid &g = c->g;
    k_sponge<T><<<grid2(g.Mloc, g.Nloc, B2D), B2D, 0, c->stream>>>(g, c->F<T>());
    note(c);
}

static void launch_dt_final(fw_ctx *c) {
    const bool d = c->p.precision == FW_PREC_FP64;
    double *dsc = d ? c->fd.dsc : c->ff.dsc;
    float *fsc = d ? c->fd.fsc : c->ff.fsc;
    unsigned long long *bits = d ? c->fd.dtmin_bits : c->ff.dtmin_bits;
    double *om = d ? c->fd.omega : c->ff.omega;
    double *cs = d ? c->fd.wmcs : c->ff.wmcs;
    float *csf = d ? c->fd.wmcsf : c->ff.wmcsf;
    k_dt_final<<<1, 128, 0, c->stream>>>(c->g, dsc, fsc, bits, om, cs, csf,
                                         c->g.wavemaker == FW_WK_JON_2D ? c->g.nfreq : 0);
    note(c);
}

template <typename T> void launch_estimate_dt(fw_ctx *c) {
    const Grid &g = c->g;
    k_dt_only<T><<<grid2(g.Mloc, g.Nloc, B2D), B2D, 0, c->stream>>>(g, c->F<T>());
    note(c);
    launch_dt_final(c);
}

template <typename T> void launch_begin_step(fw_ctx *c) {
    const Grid &g = c->g;
    const bool branch = branching(c);
    // the time step's end, which the first stage waits for before its first use
    // (join_ev), and the wavemaker's mass
    auto dt_final = [&] {
        launch_dt_final(c);
        if (branch) {
            const cudaError_t e = cudaEventRecord(c->join_ev, c->stream);
            if (e != cudaSuccess && !c->sticky_error) c->sticky_error = (int)e;
        }
        if (wm_in_band<T>(c)) {
            const int n = (g.ihi - g.ilo + 1) * (g.jhi - g.jlo + 1);
            k_wm_band<T><<<(n + 255) / 256, 256, 0, c->stream>>>(g, c->F<T>());
            note(c);
        }
    };
    if (launch_exchange_one<T, true>(c, false, B2D)) {
        on_side(c, branch, dt_final);
        return;
    }
    const int nring = 6 * g.Mloc + 6 * g.Nglob;
    k_eta0_ring<T><<<(nring + 255) / 256, 256, 0, c->stream>>>(g, c->F<T>());
    note(c);
    launch_ghost<T>(c, g.visc_breaking != 0);
    k_begin<T><<<grid2(g.Mloc, g.Nloc, B2D), B2D, 0, c->stream>>>(g, c->F<T>());
    note(c);
    on_side(c, branch, dt_final);
}

template <typename T> static void launch_disp_b(fw_ctx *c) {
    const Grid &g = c->g;
    const dim3 b = c->blk(TK_DISP_B);
    k_disp_b<T><<<grid2(g.Mloc, g.Nloc, b), b, disp_b_smem<T>(b), c->stream>>>(g, c->F<T>(), disp_k(g));
    note(c);
}
template <typename T> void launch_dispersion(fw_ctx *c) {
    launch_disp_a<T>(c);
    note(c);
    launch_disp_b<T>(c);
}

// the TMA-staged flux kernel with the maps of the current MASK buffer (its
// shared-memory size is set when the maps are made, outside any capture)
template <typename T, int DIR, int FY_> static void flux_tma_at(fw_ctx *c) {
    using S = FluxStage<T, DIR, FY_>;
    const int fi = FY_ == 8 ? 0 : (FY_ == 16 ? 1 : 2);
    const int mi = ((const void *)c->F<T>().MASK == c->fmask_base[0]) ? 0 : 1;
    k_flux_tma<T, DIR, FY_><<<flux_grid<T, DIR, FY_>(c->g), B2D, S::BYTES, c->stream>>>(c->g, c->F<T>(),
                                                                                        c->fmaps[DIR][fi][mi]);
}
template <typename T, int DIR, int FY_> bool flux_tma_attr() {
    return cudaFuncSetAttribute(k_flux_tma<T, DIR, FY_>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                FluxStage<T, DIR, FY_>::BYTES) == cudaSuccess;
}
template <typename T> bool flux_tma_attrs() {
    bool ok = flux_tma_attr<T, 0, 8>() && flux_tma_attr<T, 0, 16>() && flux_tma_attr<T, 1, 8>() &&
              flux_tma_attr<T, 1, 16>();
    if constexpr (sizeof(T) == sizeof(float)) ok = ok && flux_tma_attr<T, 0, 32>() && flux_tma_attr<T, 1, 32>();
    return ok;
}

// faces of a y strip: the busiest SM works ceil(blocks / 152) blocks of four
// strips, each with the work of about 2.3 faces before its first; in float
// a face's latency is about that of 3.5 blocks' issue, so fewer blocks than
// that on an SM gain nothing (701 x 937 FP64: 16 faces 1028 us with a third
// of the SMs idle at the end, 19 faces 680 us)
static int flux_strip(int nx, int faces, int most, bool fp64) {
    int best = 4;
    double least = 1e30;
    for (int st = 4; st <= most; st++) {
        const int blocks = nx * ((faces + 4 * st - 1) / (4 * st));
        const double cost = (st + 2.3) * std::max(fp64 ? 1.0 : 3.5, (double)((blocks + 151) / 152));
        if (cost < least) {
            least = cost;
            best = st;
        }
    }
    return best;
}

template <typename T, int DIR> static void launch_flux(fw_ctx *c) {
    const int fy = c->tune[TUNE_FLUX + DIR];
    if (c->tune[TUNE_FLUX_TMA + DIR] && c->fmaps_ok) {
        if (fy == 8) flux_tma_at<T, DIR, 8>(c);
        else if (fy == 16 || sizeof(T) == sizeof(double)) flux_tma_at<T, DIR, 16>(c);
        else if constexpr (sizeof(T) == sizeof(float)) flux_tma_at<T, DIR, 32>(c);
        note(c);
        return;
    }
    // the tuned height sets the rows of an x block and bounds the strips of y
    const Grid &g = c->g;
    const dim3 b(32, 4);
    if (DIR == 0) {
        // (more rows where the grid's blocks along y would pass the launch limit)
        const int rows = std::max({1, fy / 8, (g.Nglob + 4 * GRID_Y_MAX - 1) / (4 * GRID_Y_MAX)});
        const int nx = (g.ie + FLUX_XW) / FLUX_XW;
        k_flux_x<T><<<dim3(nx, (g.Nglob + 4 * rows - 1) / (4 * rows)), b, 0, c->stream>>>(g, c->F<T>(), rows);
    } else {
        const int nx = (g.ie + 32) / 32, strip = flux_strip(nx, g.Nglob + 1, sizeof(T) == sizeof(double) ? 2 * fy : fy, sizeof(T) == sizeof(double));
        k_flux_y<T><<<dim3(nx, (g.Nglob + 4 * strip) / (4 * strip)), b, 0, c->stream>>>(g, c->F<T>(), strip);
    }
    note(c);
}

template <typename T> static void launch_fluxes_opt(fw_ctx *c, bool branch) {
    if (branch) on_side(c, true, [&] { launch_flux<T, 1>(c); });
    launch_flux<T, 0>(c);
    if (!branch) launch_flux<T, 1>(c);
    join_side(c, branch);
}
template <typename T> void launch_fluxes(fw_ctx *c) { launch_fluxes_opt<T>(c, false); }

template <typename T> void launch_sources_debug(fw_ctx *c) {
    const Grid &g = c->g;
    k_sources<T><<<grid2(g.Mglob, g.Nglob, B2D), B2D, 0, c->stream>>>(g, c->F<T>());
    note(c);
}

// blocks of the factorisation's launch that take the reduction's multipliers
constexpr int PCR_BLOCKS = 4 * 152;
// the blocks of k_linesolve: x lines as many to a block as its threads hold,
// y columns 8 to a block, but fewer while the grid would not reach every SM
static LsfShape lsf_shape(int dir, const Grid &g, const LinePart &lp) {
    constexpr int SMS = 152;
    LsfShape S;
    const int PT = lp.P + (lp.L % LSF_M ? 1 : 0);  // threads of a line
    if (dir == 0) {
        S.nc = 1;
        S.nline = std::max(1, std::min(LSF_T / PT, (lp.nlines + SMS - 1) / SMS));
        S.nch = PT;
        S.slots = S.nline;
        S.nblk = (lp.nlines + S.nline - 1) / S.nline;
    } else {
        S.nc = PT > 128 ? 8 : PT > 64 ? 4 : PT > 32 ? 2 : 1;
        S.nline = LSF_COLS;
        if (S.nc == 1)
            while (S.nline > 2 && (g.ie + S.nline) / S.nline < SMS) S.nline /= 2;
        S.nch = (PT + S.nc - 1) / S.nc;
        // (the last chunk and its remainder rows fall into the same block: with
        // them, P is no multiple of nch for any length up to 4096)
        S.slots = S.nline / S.nc;
        S.nblk = (g.ie + S.nline) / S.nline * S.nc;  // columns 0 .. ie
    }
    // (every reduced pair has a thread too: slots x P <= nline x nch); at least
    // 128 for the staging loops
    S.nt = std::max(128, (S.nline * S.nch + 31) / 32 * 32);
    return S;
}

// The line solves' limits of shared memory.  A limit belongs to the kernel in
// this process, whatever context launches it: each is set once, when a context
// is made, to the most that any line asks for (lsf_smem_floats over all line
// lengths and counts: 62500 bytes, for x lines of 4096 rows; y 45312), and
// never to one context's own need, which would fail the launches of others.
constexpr size_t LSF_SMEM_MAX = 64 * 1024, LSX_SMEM_MAX = 200 * 1024;
template <typename T, int DIR, bool PER> static bool linesolve_attr() {
    return cudaFuncSetAttribute(k_linesolve<T, DIR, PER, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)LSF_SMEM_MAX) == cudaSuccess &&
           cudaFuncSetAttribute(k_linesolve<T, DIR, PER, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)LSF_SMEM_MAX) == cudaSuccess;
}
template <typename T> bool linesolve_attrs() {
    if constexpr (sizeof(T) == sizeof(float))
        return linesolve_attr<T, 0, false>() && linesolve_attr<T, 1, false>() && linesolve_attr<T, 1, true>() &&
               cudaFuncSetAttribute(k_linesolve_x<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)LSX_SMEM_MAX) == cudaSuccess;
    return true;
}

template <typename T, int DIR, bool PER>
static void launch_linesolve(fw_ctx *c, const LinePart &lp, bool clear_dirty) {
    const LsfShape S = lsf_shape(DIR, c->g, lp);
    auto kern = lp.L % LSF_M ? k_linesolve<T, DIR, PER, true> : k_linesolve<T, DIR, PER, false>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)S.nblk);
    cfg.blockDim = dim3((unsigned)S.nt);
    cfg.dynamicSmemBytes = lsf_smem_floats(DIR, lp, S) * sizeof(float);
    cfg.stream = c->stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)S.nc;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = S.nc > 1 ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kern, c->g, c->F<T>(), lp, S, clear_dirty ? 1 : 0);
    note(c);
}

// FP64 solves keep the factors where MASK9 stays (viscosity breaking: without
// it the wet/dry front moves MASK9, and factoring at every change would cost
// more than it saves) and tmp2 cannot vanish
static bool thomas_kept(const fw_ctx *c) {
    return c->p.precision == FW_PREC_FP64 && c->g.visc_breaking && c->g.gamma1 >= 0.0 &&
           -c->g.b1 - 2.0 * c->g.b2 >= 0.0;
}
template <typename T> static void launch_thomas_fac(fw_ctx *c) {
    const int nbx = (c->px.nlines + 31) / 32, nby = (c->py.nlines + 31) / 32;
    if (c->g.periodic) k_thomas_fac<T, true><<<nbx + nby, 32, 0, c->stream>>>(c->g, c->F<T>(), c->px, c->py, nbx);
    else k_thomas_fac<T, false><<<nbx + nby, 32, 0, c->stream>>>(c->g, c->F<T>(), c->px, c->py, nbx);
}

template <typename T, int DIR, bool PER>
static bool launch_tri(fw_ctx *c, const LinePart &lp, bool fac = true, bool clear_dirty = false) {
    const Grid &g = c->g;
    const int nt = lp.nlines * lp.P;
    if constexpr (sizeof(T) == sizeof(float)) if (c->factored) {
        if (fac) {
            k_fac_a<T, DIR, PER><<<(nt + 127) / 128, 128, 0, c->stream>>>(g, c->F<T>(), lp);
            const int nb = (lp.nlines + 127) / 128;
            const int nm = lsf_line(lp) ? std::min(lp.nlines, PCR_BLOCKS) : 0;
            k_fac_b<T, DIR, PER><<<nb + nm, 128, nm ? 12 * lp.P * sizeof(float) : 0, c->stream>>>(g, c->F<T>(), lp, nb);
            note(c, 2);
        }
        if (lsf_line(lp)) {
            launch_linesolve<T, DIR, PER>(c, lp, clear_dirty);
            return clear_dirty;
        }
        // lines of more than 4096 rows
        const size_t smem = lsx_smem_floats(lp.L, lp.P) * sizeof(float);
        if (DIR == 0 && !PER && lp.P <= 256 && smem <= LSX_SMEM_MAX) {
            k_linesolve_x<T><<<lp.nlines, 256, smem, c->stream>>>(g, c->F<T>(), lp, clear_dirty ? 1 : 0);
            note(c);
            return clear_dirty;
        }
        const dim3 gi = grid2(g.Mglob, g.Nglob, B2D);
        const int nb = std::min(512, ((2 * lp.P + 31) / 32) * 32);
        const size_t sb = (size_t)16 * lp.P * sizeof(float);
        const unsigned ga = (unsigned)((nt + 127) / 128);
        k_sol_a<T, DIR, PER, 0><<<ga, 128, 0, c->stream>>>(g, c->F<T>(), lp);
        k_sol_b<T, DIR, PER, 0><<<lp.nlines, nb, sb, c->stream>>>(g, c->F<T>(), lp);
        k_sol_c<T, DIR, 0><<<ga, 128, 0, c->stream>>>(g, c->F<T>(), lp);
        k_resid<T, DIR, PER><<<gi, B2D, 0, c->stream>>>(g, c->F<T>(), lp);
        k_sol_a<T, DIR, PER, 1><<<ga, 128, 0, c->stream>>>(g, c->F<T>(), lp);
        k_sol_b<T, DIR, PER, 1><<<lp.nlines, nb, sb, c->stream>>>(g, c->F<T>(), lp);
        k_sol_c<T, DIR, 1><<<ga, 128, 0, c->stream>>>(g, c->F<T>(), lp);
        note(c, 7);
        return false;
    }
    if constexpr (sizeof(T) == sizeof(double)) {
        if (thomas_kept(c)) {
            if (fac) {
                launch_thomas_fac<T>(c);
                note(c);
            }
            k_thomas_rhs<T, DIR, PER><<<grid2(g.Mglob, g.Nglob, B2D), B2D, 0, c->stream>>>(g, c->F<T>(), lp, clear_dirty ? 1 : 0);
            k_thomas_solve<T, DIR, PER><<<(lp.nlines + 31) / 32, dim3(32, PER ? THS_WARPS : 1), 0, c->stream>>>(g, c->F<T>(), lp);
            note(c, 2);
            return clear_dirty;
        }
        k_thomas_rows<T, DIR, PER><<<grid2(g.Mglob, g.Nglob, B2D), B2D, 0, c->stream>>>(g, c->F<T>(), lp);
        k_thomas_lines<T, DIR, PER><<<(lp.nlines + 31) / 32, 32, 0, c->stream>>>(g, c->F<T>(), lp);
        note(c, 2);
        return false;
    }
    // mixed without a constant factorisation: the partitioned solve in
    // double, one thread per chunk of m rows
    k_tri_a<T, DIR, PER><<<(nt + 127) / 128, 128, 0, c->stream>>>(g, c->F<T>(), lp);
    note(c);
    k_tri_b<T, DIR, PER><<<(lp.nlines + 127) / 128, 128, 0, c->stream>>>(g, c->F<T>(), lp);
    note(c);
    k_tri_c<T, DIR><<<(nt + 127) / 128, 128, 0, c->stream>>>(g, c->F<T>(), lp);
    note(c);
    return false;
}

// the factors that the solves of both directions keep, brought up to date when
// MASK9 has changed
template <typename T> static bool kept_factors(const fw_ctx *c) {
    return c->g.dispersion && (sizeof(T) == sizeof(float) ? c->factored != 0 : thomas_kept(c));
}
template <typename T> static void launch_factors(fw_ctx *c) {
    const Grid &g = c->g;
    if constexpr (sizeof(T) == sizeof(double)) {
        launch_thomas_fac<T>(c);
        note(c);
    } else {
        const int nbx = (c->px.nlines * c->px.P + 127) / 128;
        const int nby = (c->py.nlines * c->py.P + 127) / 128;
        const int lbx = (c->px.nlines + 127) / 128, lby = (c->py.nlines + 127) / 128;
        const int nm = std::min((lsf_line(c->px) ? c->px.nlines : 0) + (lsf_line(c->py) ? c->py.nlines : 0), PCR_BLOCKS);
        const size_t sp = nm ? 12 * std::max(lsf_line(c->px) ? c->px.P : 0, lsf_line(c->py) ? c->py.P : 0) * sizeof(float) : 0;
        if (g.periodic) {
            k_fac_a_xy<T, true><<<nbx + nby, 128, 0, c->stream>>>(g, c->F<T>(), c->px, c->py, nbx);
            k_fac_b_xy<T, true><<<lbx + lby + nm, 128, sp, c->stream>>>(g, c->F<T>(), c->px, c->py, lbx, lby);
        } else {
            k_fac_a_xy<T, false><<<nbx + nby, 128, 0, c->stream>>>(g, c->F<T>(), c->px, c->py, nbx);
            k_fac_b_xy<T, false><<<lbx + lby + nm, 128, sp, c->stream>>>(g, c->F<T>(), c->px, c->py, lbx, lby);
        }
        note(c, 2);
    }
}

// ESTIMATE_HUV; with_post = false leaves the GET_Eta_U_V_HU_HV tail (k_post)
// to the fused kernel of the stage; branch: a captured stage, whose side branch
// has brought the factors up to date and is joined
template <typename T> static void launch_estimate_huv_opt(fw_ctx *c, int istage, bool with_post, bool branch) {
    const Grid &g = c->g;
    static const double AL[3] = {0.0, 3.0 / 4.0, 1.0 / 3.0};
    static const double BE[3] = {1.0, 1.0 / 4.0, 2.0 / 3.0};
    const T al = (T)AL[istage - 1], be = (T)BE[istage - 1];
    // stage 2 too: with PERIODIC, EXCHANGE leaves the x-ghost values of the
    // previous exchange in the ghost corners (bc.F:735-740), so the last
    // stage's corners hold the second stage's values
    if (istage >= 2 && g.track_rad)
        launch_update<T, true>(c, al, be, wm_in_band<T>(c));
    else
        launch_update<T, false>(c, al, be, wm_in_band<T>(c));
    note(c);
    if (g.dispersion) {
        if (!branch && kept_factors<T>(c)) launch_factors<T>(c);
        auto y = [&] {
            if (g.periodic) launch_tri<T, 1, true>(c, c->py, false);
            else launch_tri<T, 1, false>(c, c->py, false);
        };
        if (sizeof(T) == sizeof(float) && c->factored) {
            // the x solve resets the change flag when it can
            const bool both = branch && lsf_line(c->px) && lsf_line(c->py);
            if (both) on_side(c, true, y);
            const bool cleared = launch_tri<T, 0, false>(c, c->px, false, true);
            if (!both) y();
            join_side(c, both);
            if (!cleared) {
                k_fac_clear<<<1, 1, 0, c->stream>>>(c->F<T>().m9_dirty);
                note(c);
            }
        } else {
            // (the x solve clears the change flag of kept FP64 factors)
            const bool kept = kept_factors<T>(c), both = branch && kept;
            if (both) on_side(c, true, y);
            launch_tri<T, 0, false>(c, c->px, !kept, true);
            if (!both) y();
            join_side(c, both);
        }
    }
    if (!with_post) return;
    k_post<T><<<grid2(g.Mloc, g.Nloc, B2D), B2D, 0, c->stream>>>(g, c->F<T>());
    note(c);
    if (!g.dispersion) {
        k_nodisp_copy<T><<<grid2(g.Mloc, g.Nloc, B2D), B2D, 0, c->stream>>>(g, c->F<T>());
        note(c);
    }
}

template <typename T> void launch_estimate_huv(fw_ctx *c, int istage) { launch_estimate_huv_opt<T>(c, istage, true, false); }

template <typename T> void launch_update_mask(fw_ctx *c) {
    const Grid &g = c->g;
    k_mask<T><<<grid2(g.Mloc + 1, g.Nloc + 1, B2D), B2D, 0, c->stream>>>(g, c->F<T>());
    note(c);
    auto &F = c->F<T>();
    uint8_t *t = F.MASK;
    F.MASK = F.MASKn;
    F.MASKn = t;
}

template <typename T> void launch_breaking(fw_ctx *c) {
    const Grid &g = c->g;
    if (!g.show_breaking) return;
    k_break_a<T><<<grid2(g.Mloc, g.Nloc, B2D), B2D, 0, c->stream>>>(g, c->F<T>());
    note(c);
    k_break_b<T><<<1, 1024, 0, c->stream>>>(g, c->F<T>());
    note(c);
    auto &F = c->F<T>();
    T *t = F.AGE;
    F.AGE = F.AGEn;
    F.AGEn = t;
}

// CALCULATE_Cm_Sm (wavemaker.F:831-891) on the wavemaker band: one thread
// per (band cell, frequency) sums the Ntheta directional components
//   Cm/Sm = sum_kt D_gen(kf,kt) exp(-beta_gen(kf) ((I-Ibeg) DX - Xc)^2)
//           cos/sin(rlamda(kf,kt) (J-Jbeg) DY + phi1(kf,kt))
// in double, in the reference's order, and stores it in the field precision.
// i0, j0: I-Ibeg and J-Jbeg of the band's first cell.
template <typename T>
__global__ void __launch_bounds__(256) k_cm_sm(int bw, int bh, int mf, int mt, int i0, int j0, double DX,
                                               double DY, double xc, const double *__restrict__ tab, T *Cm,
                                               T *Sm) {
    const long long nb = (long long)bw * bh;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nb * mf) return;
    const int kf = (int)(t / nb);
    const long long b = t - (long long)kf * nb;
    const int bj = (int)(b / bw), bi = (int)(b - (long long)bj * bw);
    const double *dgen = tab, *rlamda = tab + (size_t)mf * mt, *phi = tab + 2 * (size_t)mf * mt;
    const double *betagen = tab + 3 * (size_t)mf * mt;
    const double dx = (double)(i0 + bi) * DX - xc;
    const double y = (double)(j0 + bj) * DY - 0.0;
    const double ex = exp(-betagen[kf] * (dx * dx));
    double cm = 0.0, sm = 0.0;
    for (int kt = 0; kt < mt; kt++) {
        const size_t k2 = (size_t)kf + (size_t)kt * mf;
        const double amp = dgen[k2] * ex;
        const double arg = rlamda[k2] * y + phi[k2];
        cm = cm + amp * cos(arg);
        sm = sm + amp * sin(arg);
    }
    Cm[b + (size_t)kf * nb] = (T)cm;
    Sm[b + (size_t)kf * nb] = (T)sm;
}

template <typename T>
void launch_cm_sm(fw_ctx *c, int bw, int bh, int i0, int j0, const double *tab, T *Cm, T *Sm) {
    const Grid &g = c->g;
    const long long n = (long long)bw * bh * g.nfreq;
    k_cm_sm<T><<<(unsigned)((n + 255) / 256), 256, 0, c->stream>>>(bw, bh, g.nfreq, c->p.ntheta, i0, j0, g.DX,
                                                                   g.DY, g.xc_wk, tab, Cm, Sm);
    note(c);
}

template <typename T> void launch_end_step(fw_ctx *c) {
    const Grid &g = c->g;
    if (g.stats) {
        k_tsum<<<1, 1, 0, c->stream>>>(g, c->F<T>().dsc, c->F<T>().fsc);
        note(c);
    }
    k_end<T><<<grid2(g.Mloc, g.Nloc, B2D), B2D, 0, c->stream>>>(g, c->F<T>(), c->p.track_hmax);
    note(c);
    if (g.track_rad) {
        k_rad_derived<T><<<grid2(g.ie - g.ib + 1, g.je - g.jb + 1, B2D), B2D, 0, c->stream>>>(g, c->F<T>());
        note(c);
    }
}

template <typename T> void launch_stage(fw_ctx *c, int istage) {
    const Grid &g = c->g;
    const bool branch = branching(c);
    if (branch && kept_factors<T>(c)) on_side(c, true, [&] { launch_factors<T>(c); });
    if (g.dispersion) {
        launch_disp_a<T>(c);
        note(c);
    }
    if (branch && istage == 1) {
        const cudaError_t e = cudaStreamWaitEvent(c->stream, c->join_ev, 0);
        if (e != cudaSuccess && !c->sticky_error) c->sticky_error = (int)e;
    }
    if (g.dispersion) launch_disp_b<T>(c);
    launch_fluxes_opt<T>(c, branch);
    if (g.dispersion && g.show_breaking) {
        // GET_Eta_U_V_HU_HV tail + UPDATE_MASK + BREAKING (parallel part)
        // in one kernel, then the breaking sweep's candidates
        launch_estimate_huv_opt<T>(c, istage, false, branch);
        launch_pmb<T>(c);
        note(c);
        auto &F = c->F<T>();
        uint8_t *t = F.MASK;
        F.MASK = F.MASKn;
        F.MASKn = t;
        k_break_b<T><<<1, 1024, 0, c->stream>>>(g, F);
        note(c);
        T *a = F.AGE;
        F.AGE = F.AGEn;
        F.AGEn = a;
    } else {
        launch_estimate_huv_opt<T>(c, istage, true, branch);
        launch_update_mask<T>(c);
        launch_breaking<T>(c);
    }
    launch_exchange<T>(c, g.direct_sponge != 0);
    if (istage >= 2 && g.track_rad) {
        const int n = 6 * g.Nglob + 6 * g.Mloc;
        k_ghost_rad<T><<<(n + 255) / 256, 256, 0, c->stream>>>(g, c->F<T>());
        note(c);
    }
}

#ifdef FW_SHARED_DEFS
// ---------------------------------------------------------------------------
// host-layout conversion: a Fortran (w x h, leading dimension w) array in a
// device staging buffer <-> a pitched field
// ---------------------------------------------------------------------------
template <typename S, typename D>
__global__ void k_unpack(const S *src, int w, int h, D *dst, int pitch) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= w || j >= h) return;
    dst[(size_t)i + (size_t)j * pitch] = (D)src[(size_t)i + (size_t)j * w];
}
template <typename S, typename D>
__global__ void k_pack(const S *src, int pitch, int w, int h, D *dst) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= w || j >= h) return;
    dst[(size_t)i + (size_t)j * w] = (D)src[(size_t)i + (size_t)j * pitch];
}
__global__ void k_unpack_mask(const int *src, int w, int h, uint8_t *dst, int pitch) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= w || j >= h) return;
    const int v = src[(size_t)i + (size_t)j * w];
    dst[(size_t)i + (size_t)j * pitch] = (uint8_t)(v > 0 ? 1 : 0);
}

void convert_in(fw_ctx *c, const void *staging, int is_mask, void *field, int w, int h) {
    const dim3 b(32, 8), gr((w + 31) / 32, (h + 7) / 8);
    if (is_mask) k_unpack_mask<<<gr, b, 0, c->stream>>>((const int *)staging, w, h, (uint8_t *)field, c->g.pitch);
    else k_unpack<double, float><<<gr, b, 0, c->stream>>>((const double *)staging, w, h, (float *)field, c->g.pitch);
    note(c);
}
void convert_out(fw_ctx *c, const void *field, int is_mask, void *staging, int w, int h) {
    const dim3 b(32, 8), gr((w + 31) / 32, (h + 7) / 8);
    if (is_mask) k_pack<uint8_t, int><<<gr, b, 0, c->stream>>>((const uint8_t *)field, c->g.pitch, w, h, (int *)staging);
    else k_pack<float, double><<<gr, b, 0, c->stream>>>((const float *)field, c->g.pitch, w, h, (double *)staging);
    note(c);
}

// float host arrays (an FP32 host's REAL(SP) fields) of the FP64 build:
// widened on the way in, rounded to nearest on the way out
void convert_in_f32(fw_ctx *c, const float *staging, double *field, int w, int h) {
    const dim3 b(32, 8), gr((w + 31) / 32, (h + 7) / 8);
    k_unpack<float, double><<<gr, b, 0, c->stream>>>(staging, w, h, field, c->g.pitch);
    note(c);
}
void convert_out_f32(fw_ctx *c, const double *field, float *staging, int w, int h) {
    const dim3 b(32, 8), gr((w + 31) / 32, (h + 7) / 8);
    k_pack<double, float><<<gr, b, 0, c->stream>>>(field, c->g.pitch, w, h, staging);
    note(c);
}

// values of one field at n cells (pitched offsets) as double; type 0 double,
// 1 float, 2 uint8 mask
__global__ void k_gather(const void *field, int type, const int *off, int n, double *out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int o = off[k];
    out[k] = type == 0 ? ((const double *)field)[o]
                       : type == 1 ? (double)((const float *)field)[o] : (double)((const uint8_t *)field)[o];
}
void gather_points(fw_ctx *c, const void *field, int type, const int *d_off, int n, double *d_out) {
    k_gather<<<(n + 127) / 128, 128, 0, c->stream>>>(field, type, d_off, n, d_out);
    note(c);
}

#endif  // FW_SHARED_DEFS

// one kernel of the step by name, for timing (fw_time_kernel)
template <typename T> int launch_by_name(fw_ctx *c, const char *name) {
    const Grid &g = c->g;
    Fields<T> &f = c->F<T>();
    const dim3 gc = grid2(g.Mloc, g.Nloc, B2D);
    auto is = [&](const char *n) { return std::strcmp(name, n) == 0; };
    if (is("disp_a")) launch_disp_a<T>(c);
    else if (is("disp_b")) { launch_disp_b<T>(c); return 0; }
    else if (is("flux_x")) { launch_flux<T, 0>(c); return 0; }
    else if (is("flux_y")) { launch_flux<T, 1>(c); return 0; }
    else if (is("update")) launch_update<T, false>(c, (T)0.75, (T)0.25, wm_has_band<T>(c));  // as in a whole step
    else if (is("post_mask_break")) launch_pmb<T>(c);
    else if (is("tri_x")) { launch_tri<T, 0, false>(c, c->px); return 0; }
    else if (is("tri_y")) {
        if (g.periodic) launch_tri<T, 1, true>(c, c->py);
        else launch_tri<T, 1, false>(c, c->py);
        return 0;
    }
    else if (is("post")) k_post<T><<<gc, B2D, 0, c->stream>>>(g, f);
    else if (is("mask")) k_mask<T><<<grid2(g.Mloc + 1, g.Nloc + 1, B2D), B2D, 0, c->stream>>>(g, f);
    else if (is("break_a")) k_break_a<T><<<gc, B2D, 0, c->stream>>>(g, f);
    else if (is("ghost")) { launch_ghost<T>(c, g.visc_breaking != 0); return 0; }
    else if (is("maskmul") && launch_exchange_one<T, false>(c, g.direct_sponge, c->blk(TK_MASKMUL))) return 0;
    else if (is("begin") && launch_exchange_one<T, true>(c, false, B2D)) return 0;
    else if (is("maskmul")) k_maskmul<T><<<grid2(g.Mloc, g.Nloc, c->blk(TK_MASKMUL)), c->blk(TK_MASKMUL), 0, c->stream>>>(g, f, g.direct_sponge);
    else if (is("begin")) k_begin<T><<<gc, B2D, 0, c->stream>>>(g, f);
    else return -1;
    note(c);
    return 0;
}

#define INST(T)                                                  \
    template void launch_begin_step<T>(fw_ctx *);                \
    template void launch_exchange<T>(fw_ctx *, bool);            \
    template void launch_estimate_dt<T>(fw_ctx *);               \
    template void launch_dispersion<T>(fw_ctx *);                \
    template void launch_fluxes<T>(fw_ctx *);                    \
    template void launch_sources_debug<T>(fw_ctx *);             \
    template void launch_estimate_huv<T>(fw_ctx *, int);         \
    template void launch_update_mask<T>(fw_ctx *);               \
    template void launch_breaking<T>(fw_ctx *);                  \
    template void launch_sponge<T>(fw_ctx *);                    \
    template void launch_end_step<T>(fw_ctx *);                  \
    template void launch_stage<T>(fw_ctx *, int);     \
    template void launch_cm_sm<T>(fw_ctx *, int, int, int, int, const double *, T *, T *); \
    template int launch_by_name<T>(fw_ctx *, const char *);      \
    template bool flux_tma_attrs<T>();                           \
    template bool linesolve_attrs<T>();

}  // namespace fw
