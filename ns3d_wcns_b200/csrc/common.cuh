// common.cuh -- device layout and the exact-rounding state conversions shared
// by every kernel of the B200 ns3d_wcns path.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace ns3d {

constexpr int NG = 3;  // ghost layers for WENO5/MDCD (initialization.cpp:175-192)
constexpr int CHIP_SMS = 148;  // B200: what the rules that split the work by size count on

// Padded device layout of one Field3D array: element (i,j,k), i in [0,sx),
// lives at ((k*sy + j)*px + i + off).  off puts the first interior cell
// (i = 3) on a 32-byte sector boundary; px keeps every row sector aligned.
struct Layout {
    int nx, ny, nz;     // interior
    int sx, sy, sz;     // with ghosts
    int px, off;        // pitch and x offset (elements)
    long plane;         // elements of one padded array (sz*sy*px, rounded)
    __host__ __device__ __forceinline__ long at(int i, int j, int k) const {
        return ((long)k * sy + j) * px + i + off;
    }
};

template <typename T>
inline Layout make_layout(int nx, int ny, int nz) {
    Layout L;
    L.nx = nx; L.ny = ny; L.nz = nz;
    L.sx = nx + 2 * NG; L.sy = ny + 2 * NG; L.sz = nz + 2 * NG;
    const int per_sector = 32 / (int)sizeof(T);
    L.off = per_sector - NG;  // (NG + off) * sizeof(T) == 32
    L.px = ((L.sx + L.off + per_sector - 1) / per_sector) * per_sector;
    long n = (long)L.sz * L.sy * L.px;
    const long align = 256 / (long)sizeof(T);
    L.plane = ((n + align - 1) / align) * align;
    return L;
}

// Device-resident time-advance state (the dt schedule of time_advance,
// maincycle.cpp:18-56, run on the device so that many steps need no host
// round trip).  While `done` is set every kernel of a step returns at once.
struct DevClock {
    double t, dt, t_end, cfl_min;
    int done, steps, budget, err;
};

// Physical constants (initialization.cpp:194-197, field_structures.h:95).
struct Phys {
    double gamma, Rgas, Cp, Pr, mu, S;
    double inv_dx, inv_dy, inv_dz;
    double dx, dy, dz;
    double mdcd_disp, mdcd_diss;
};

// ---------------------------------------------------------------------------
// FP64 reciprocal, square root and quotient for the kernels' inner loops.
// A hardware seed (rcp / rsqrt.approx.ftz.f64, about 20 bits) and one
// third-order iteration (Householder's method: with e = 1 - x y,
// 1/x = y (1 + e + e^2 + ...); with r = 1 - t y^2,
// sqrt(t) = t y (1 + r/2 + 3 r^2/8 + ...)) leave a truncation error below
// 2^-57, so the result is within 0.6 ulp (reciprocal) and 0.8 ulp (square
// root).  Three and five FP64 instructions without a branch, against the
// IEEE operations' seven to ten with their range checks and slow paths; the
// sweeps hold five to thirteen of them per face (256^3, x-sweep: 0.900 -> 0.826 ms
// with MDCD_HYBRID + HLLC, 1.338 -> 1.207 with WENO5 + Roe).  Range: x normal with a
// normal reciprocal (zero, subnormal and infinite x give NaN, x above 2^1022
// gives 0); sqrt_fp64 returns 0 for zero and subnormal arguments and NaN for
// negative and infinite ones.  In a face's flux these stand for states that the
// scheme has no finite flux for; the conversions below look for them.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double rcp_fp64(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = __fma_rn(-x, y, 1.0);
    return __fma_rn(y, __fma_rn(e, e, e), y);
}
__device__ __forceinline__ double sqrt_fp64(double t) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(t));
    const double a = t * y, r = __fma_rn(-a, y, 1.0);
    const double s = __fma_rn(a * r, __fma_rn(r, 0.375, 0.5), a);
    return fabs(t) < 2.2250738585072014e-308 ? 0.0 : s;
}
// a / b from y = rcp_fp64(b): one reciprocal serves several quotients of the
// same divisor.  The residual of the first quotient is exact in one FMA, and
// the corrected quotient is off by 2^-103 of itself before it is rounded
// (P. W. Markstein, IBM J. Res. Dev. 34 (1990) 111, whose theorem asks for a
// correctly rounded y): the IEEE quotient, but for one that close to a tie.
// Zeros keep their sign for b > 0.  Not for what rcp_fp64 excludes, quotients
// that overflow (NaN), and numerators below 2^-960 (the residual underflows).
__device__ __forceinline__ double div_fp64(double a, double b, double y) {
    const double q = a * y;
    return __fma_rn(-__fma_rn(q, b, -a), y, q);
}

// Neither infinite nor NaN.  An integer test: the FP64 pipe is what the sweeps wait for.
__device__ __forceinline__ bool finite_fp64(double x) { return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000; }
// The IEEE quotient out of line: for branches that no ordinary state takes, in
// kernels that fill the instruction cache.
static __device__ __noinline__ double div_ieee(double a, double b) { return __ddiv_rn(a, b); }

// ---------------------------------------------------------------------------
// Conversions with the reference's rounding.  The reference compiles without
// fused multiply-add, so these use the _rn intrinsics (no contraction) and
// div_fp64.  Where the result is not finite the IEEE operations decide (a branch
// that no ordinary state takes), so zero, subnormal and infinite divisors and
// overflows give what they give there.  ENDS: 1 with that branch, 0 without it
// (the stencils of the sweeps, which have no finite flux for such a state, and
// fused_stage_cell, which asks once for all its conversions), 2 the IEEE
// operations.  A branch in each cost the 192^3 x- and z-sweeps 1.5 and 3 %.
// ---------------------------------------------------------------------------
template <int ENDS>
__device__ __forceinline__ double div_ends(double a, double b, double y) {
    return ENDS == 2 ? div_ieee(a, b) : div_fp64(a, b, y);
}

// Field3D::primitiveToConserved, field_structures.h:468-488.
template <int ENDS = 1>
__device__ __forceinline__ void p2c_exact(double r, double u, double v, double w, double p, double gamma,
                                          double U[5]) {
    double rr = r <= 0.0 ? 1e-12 : r;
    U[0] = rr;
    U[1] = __dmul_rn(rr, u);
    U[2] = __dmul_rn(rr, v);
    U[3] = __dmul_rn(rr, w);
    double kin = __dmul_rn(0.5, __dadd_rn(__dadd_rn(__dmul_rn(u, u), __dmul_rn(v, v)), __dmul_rn(w, w)));
    const double d = __dmul_rn(gamma - 1.0, rr);
    double e = div_ends<ENDS>(p, d, rcp_fp64(d));
    U[4] = __dmul_rn(rr, __dadd_rn(e, kin));
    if (ENDS == 1 && __builtin_expect(!finite_fp64(U[4]), 0)) U[4] = __dmul_rn(rr, __dadd_rn(div_ieee(p, d), kin));
}

// Field3D::conservedToPrimitive, field_structures.h:444-465 (density clamp).
template <int ENDS = 1>
__device__ __forceinline__ void c2p_exact(const double U[5], double gamma, double W[5]) {
    double rr = U[0] <= 0.0 ? 1e-12 : U[0];
    const double ir = rcp_fp64(rr);
    double u = div_ends<ENDS>(U[1], rr, ir), v = div_ends<ENDS>(U[2], rr, ir), w = div_ends<ENDS>(U[3], rr, ir);
    double kin = __dmul_rn(0.5, __dadd_rn(__dadd_rn(__dmul_rn(u, u), __dmul_rn(v, v)), __dmul_rn(w, w)));
    double e = __dsub_rn(div_ends<ENDS>(U[4], rr, ir), kin);
    W[0] = rr; W[1] = u; W[2] = v; W[3] = w;
    W[4] = __dmul_rn(__dmul_rn(gamma - 1.0, rr), e);
    if constexpr (ENDS == 1) {
        if (__builtin_expect(!finite_fp64(W[4]), 0)) c2p_exact<2>(U, gamma, W);
    }
}

// T = p / (rho Rgas), field_structures.h:486
template <int ENDS = 1>
__device__ __forceinline__ double temperature_exact(const double W[5], double Rgas) {
    const double d = __dmul_rn(W[0], Rgas);
    double T = div_ends<ENDS>(W[4], d, rcp_fp64(d));
    if (ENDS == 1 && __builtin_expect(!finite_fp64(T), 0)) T = div_ieee(W[4], d);
    return T;
}

// Mixed path: conserved -> primitive in FP64 with one reciprocal (the mixed
// path has an accuracy bound, not a bitwise contract); the pressure
// recovery p = (gamma-1)(E - rho |u|^2 / 2), which cancels at low Mach, stays
// FP64.  Density clamp as field_structures.h:444-465.
__device__ __forceinline__ void c2p_fast(const double U[5], double gamma, double W[5], double &irho) {
    const double rr = U[0] <= 0.0 ? 1e-12 : U[0];
    irho = 1.0 / rr;
    const double u = U[1] * irho, v = U[2] * irho, w = U[3] * irho;
    W[0] = rr; W[1] = u; W[2] = v; W[3] = w;
    W[4] = (gamma - 1.0) * (U[4] - 0.5 * rr * (u * u + v * v + w * w));
}

// Float versions for the mixed path (no parity contract).
__device__ __forceinline__ void p2c_f(float r, float u, float v, float w, float p, float gm1,
                                      float U[5]) {
    float rr = r <= 0.f ? 1e-12f : r;
    U[0] = rr; U[1] = rr * u; U[2] = rr * v; U[3] = rr * w;
    U[4] = p / gm1 + 0.5f * rr * (u * u + v * v + w * w);
}

}  // namespace ns3d

namespace ns3d {
// Asynchronous global -> shared copies (LDGSTS), used to stage the next chunk
// of a sweep while the current one computes.
__device__ __forceinline__ void cp_async(double *smem_dst, const double *gsrc) {
    unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async(float *smem_dst, const float *gsrc) {
    unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }
}  // namespace ns3d
