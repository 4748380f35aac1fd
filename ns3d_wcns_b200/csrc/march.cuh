// march.cuh -- the component-wise sweeps along y and z, one line per thread.
//
// The work of sweep_kernel (sweep.cuh): primitive -> conserved, WCNS
// interpolation, Riemann flux, the half-node ghost faces, the 6th-order
// half-node difference, this direction's viscous divergence and, along z, the
// fused RK stage.  The unit of work differs.  A thread owns one line (mixed
// path: two x-neighbouring lines in the halves of a float2) and walks it cell
// by cell.  The six-cell stencil of conserved states and the last faces slide
// through registers; the line's node viscous fluxes, the next cell, the old
// right-hand side and the step-start state arrive by cp.async in slots of
// shared memory that only this thread reads.  So nothing in the loop waits on
// another thread: no block barriers, no tails to move, each cell's detector
// evaluated once, and every stencil value is a register.
//
// Lines are numbered across the whole plane (x fastest), so a warp is full
// whatever nx is and its accesses stay contiguous.  A line is cut into
// segments (gridDim.y) when there are too few lines to fill the chip; a
// segment recomputes the five faces it shares with its neighbours.
//
// 256^3, one launch, against the chunked kernel (a face per thread, shared
// stencils, three barriers a chunk) that it replaced: FP64 MDCD_HYBRID + HLLC y
// 0.861 -> 0.703 ms, fused z 1.127 -> 0.917; WENO5 + Roe 1.222 -> 0.892 and 1.512
// -> 1.10; mixed 0.431 -> 0.372 and 0.672 -> 0.623.  Issue and FP64 latency
// bound it now: 11 warps per SM (162-168 registers), issue slots 48-55 % and the
// FP64 pipe 39-43 % busy, 3.4 TB/s.
#pragma once

#include "pair.cuh"

namespace ns3d {

constexpr int MARCH_NT = 64;  // threads per block (no cooperation between its warps)

template <typename T>
struct LaneOf {
    using R = T;
    static constexpr int N = 1;
};
template <>
struct LaneOf<float2> {
    using R = float;
    static constexpr int N = 2;
};

template <typename T>
struct MarchArgs {
    SweepArgs<typename LaneOf<T>::R> a;
    T lin[6];        // MDCD linear coefficients (both halves for float2)
    T dc[3], inv_h;  // half-node difference (SweepArgs)
    T vc[3], inv_60h;  // 6th-order derivative
    int nlines;      // line units: lines (pairs of lines for float2) of the swept planes
    int seg_len;     // cells per segment
};

// ---------------------------------------------------------------- one value

__device__ __forceinline__ void march_cons(double gamma, const double *w, double *U) {
    p2c_exact<0>(w[0], w[1], w[2], w[3], w[4], gamma, U);
}
__device__ __forceinline__ void march_cons(float gamma, const float *w, float *U) {
    p2c_f(w[0], w[1], w[2], w[3], w[4], gamma - 1.f, U);
}
__device__ __forceinline__ void march_cons(float gamma, const float2 *w, float2 *U) {
    float a[5], b[5];
    p2c_f(w[0].x, w[1].x, w[2].x, w[3].x, w[4].x, gamma - 1.f, a);
    p2c_f(w[0].y, w[1].y, w[2].y, w[3].y, w[4].y, gamma - 1.f, b);
#pragma unroll
    for (int q = 0; q < 5; ++q) U[q] = make_float2(a[q], b[q]);
}

// rounded on its own: the same bits from every copy of the boundary code
__device__ __forceinline__ double march_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float march_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float2 march_add(float2 a, float2 b) { return add2(a, b); }
template <typename R, typename F>
__device__ __forceinline__ R march_visc_edge(R, F v, int order, const R *dinv) {
    return dstencil_inv<R>(v, order, dinv);
}
template <typename F>
__device__ __forceinline__ float2 march_visc_edge(float2, F v, int order, const float *dinv) {
    return make_float2(dstencil_inv<float>([&](int o) { return v(o).x; }, order, dinv),
                       dstencil_inv<float>([&](int o) { return v(o).y; }, order, dinv));
}

template <typename T>
__device__ __forceinline__ T march_const(double v) { return (T)v; }
template <>
__device__ __forceinline__ float2 march_const<float2>(double v) { return p2((float)v); }

// line h of a value
__device__ __forceinline__ float march_half(float v, int) { return v; }
__device__ __forceinline__ float march_half(float2 v, int h) { return h ? v.y : v.x; }
__device__ __forceinline__ void march_set(float &v, int, float x) { v = x; }
__device__ __forceinline__ void march_set(float2 &v, int h, float x) { if (h) v.y = x; else v.x = x; }
__device__ __forceinline__ double march_half(double v, int) { return v; }
__device__ __forceinline__ void march_set(double &v, int, double x) { v = x; }
__device__ __forceinline__ void march_cp(double *dst, const double *src) { cp_async(dst, src); }
__device__ __forceinline__ void march_cp(float *dst, const float *src) { cp_async(dst, src); }
__device__ __forceinline__ void march_cp(float2 *dst, const float *src) { cp_async8(dst, src); }
template <typename T, typename R>
__device__ __forceinline__ T march_ld(const R *p) { return *reinterpret_cast<const T *>(p); }

// ------------------------------------------------------------------ one face

// Whether the detector of one cell does not clearly accept the linear scheme
// for one variable, from its five points (bit 0; bit 5 for a float2's second
// line).  FP64: the two sides of the cross-multiplied test (mdcd_smooth, both
// scaled by 5/2) compared by their high words; anything rejected or closer
// than two units in them is left to march_weno, which takes mdcd_smooth's
// decision.
__device__ __forceinline__ unsigned march_doubt1(double f0, double f1, double f2, double f3, double f4) {
    const double eps = 0.9 * 0.4 / (1.0 - 0.9 * 0.4) * 1e-4;
    const double a = fabs(f2 - f1) + fabs(f2 - 2.0 * f1 + f0);
    const double b = fabs(f2 - f3) + fabs(f2 - 2.0 * f3 + f4);
    const double lhs = __fma_rn(5.0 * a, b, 2.5 * eps), rhs = __fma_rn(a, a, __fma_rn(b, b, eps));
    return f64_hi_word(lhs) - f64_hi_word(rhs) <= 1 ? 1u : 0u;
}
__device__ __forceinline__ unsigned march_doubt1(float f0, float f1, float f2, float f3, float f4) {
    return mdcd_smooth(f0, f1, f2, f3, f4) ? 0u : 1u;
}
__device__ __forceinline__ unsigned march_doubt1(float2 f0, float2 f1, float2 f2, float2 f3, float2 f4) {
    bool sa, sb;
    mdcd_smooth2(f0, f1, f2, f3, f4, sa, sb);
    return (sa ? 0u : 1u) | (sb ? 0u : 32u);
}
template <typename T>
__device__ __forceinline__ unsigned march_doubt1(const T *f) { return march_doubt1(f[0], f[1], f[2], f[3], f[4]); }
// every variable: bit q (and q + 5); u[m][q]
template <typename T>
__device__ __forceinline__ unsigned march_doubt(const T (*u)[5]) {
    unsigned r = 0;
#pragma unroll
    for (int q = 0; q < 5; ++q) r |= march_doubt1(u[0][q], u[1][q], u[2][q], u[3][q], u[4][q]) << q;
    return r;
}

// Position of the nth set bit (nth < popc(mask)).
__device__ __forceinline__ int march_nth_bit(unsigned mask, int nth) {
    int pos = 0;
#pragma unroll
    for (int s = 16; s; s >>= 1) {
        const int c = __popc((mask >> pos) & ((1u << s) - 1u));
        if (nth >= c) { nth -= c; pos += s; }
    }
    return pos;
}
__device__ __forceinline__ double march_shfl(double v, int src, int) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ float march_shfl(float v, int src, int) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ float march_shfl(float2 v, int src, int line) {
    const float x = __shfl_sync(0xffffffffu, v.x, src), y = __shfl_sync(0xffffffffu, v.y, src);
    return line ? y : x;
}

// WENO states from the stencil g of a face: one side (right: from the reversed
// stencil) into a, or both, the right one into b, through one copy of the code.
// keep: the linear states stay (the reversed stencil gives the same decision).
template <typename R, typename H>
__device__ __forceinline__ void march_sides(const H &hd, bool both, bool right, const R *g, R &a, R &b, bool &keep) {
    keep = false;
    if constexpr (sizeof(R) == 8)
        keep = mdcd_smooth(g[0], g[1], g[2], g[3], g[4]) && mdcd_smooth(g[1], g[2], g[3], g[4], g[5]);
    a = b = R(0);
    bool rev = right && !both;
#pragma unroll 1
    for (int e = 0; e <= (both ? 1 : 0); ++e) {
        const R s = mdcd_weno_branch(hd, rev ? g[5] : g[0], rev ? g[4] : g[1], rev ? g[3] : g[2], rev ? g[2] : g[3],
                                     rev ? g[1] : g[4], rev ? g[0] : g[5]);
        if (e == 0) a = s;
        else b = s;
        rev = true;
    }
}

// The states of the variables in doubt, for a warp in which some lane has
// one: every (lane, variable, line) in doubt is a task, the tasks are dealt
// out over pairs of lanes, one for each side, or, where they are more than
// sixteen, over the lanes; a lane fetches its stencil by shuffles, takes the
// exact decision (FP64) and evaluates its side or sides, and the results go
// back.  An under-resolved flow has a
// few tasks at most faces (64^3 decaying turbulence: 2.6 on average, some at
// 87 % of the faces); one round then replaces a divergent branch per variable
// and side, which the whole warp would walk through (y-sweep there: 60 -> 41 us
// with both sides always in one lane; with the segments of today 50 -> 43 us
// from that to this, z 55 -> 48, 96^3 x / y / z 76 / 92 / 105 -> 72 / 78 / 91, mixed
// 128^3 90 / 91 / 137 -> 87 / 82 / 123; a flow with more than sixteen at most
// faces, 64^3 later on, keeps its time, where sixteen at a time cost 8 % more).
template <typename T>
__device__ __forceinline__ void march_weno(const MarchArgs<T> &m, const T (*u)[5], unsigned doubt, T *UL, T *UR) {
    using R = typename LaneOf<T>::R;
    constexpr int NV = 5 * LaneOf<T>::N;
    const int lane = threadIdx.x & 31;
    int total = 0;
#pragma unroll
    for (int v = 0; v < NV; ++v) total += __popc(__ballot_sync(0xffffffffu, (doubt >> v) & 1u));
    int base = 0;
#pragma unroll 1
    do {
        const bool both = total - base > 16;
        const int sh = both ? 0 : 1, width = 32 >> sh;  // lanes per task, tasks of the round
        int var = -1, nth = 0, off = base + (lane >> sh);  // this lane's task
        unsigned mask = 0;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const unsigned b = __ballot_sync(0xffffffffu, (doubt >> v) & 1u);
            const int c = __popc(b);
            if (off >= 0 && off < c) { var = v; mask = b; nth = off; }
            off -= c;
        }
        const int src = march_nth_bit(mask, nth) & 31, line = var >= 5, q0 = line ? var - 5 : var;
        R g[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) g[k] = R(0);
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            if (!__any_sync(0xffffffffu, q0 == q)) continue;
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                const R x = march_shfl(u[k][q], src, line);
                if (q0 == q) g[k] = x;
            }
        }
        bool keep;
        R sa, sb;
        march_sides(m.a.sp.hd, both, (lane & 1) != 0, g, sa, sb, keep);
        if (!both) sb = sa;
        int from = -base;  // the task of this lane's variable v is number `from` + its rank of the round
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const unsigned b = __ballot_sync(0xffffffffu, (doubt >> v) & 1u);
            if (!b) continue;
            const int t = from + __popc(b & ((1u << lane) - 1u));
            const int at = (t << sh) & 31;
            const R lv = __shfl_sync(0xffffffffu, sa, at), rv = __shfl_sync(0xffffffffu, sb, at + sh);
            const bool kv = __shfl_sync(0xffffffffu, (int)keep, at);
            if (((doubt >> v) & 1u) && t >= 0 && t < width && !kv) {
                march_set(UL[v % 5], v / 5, lv);
                march_set(UR[v % 5], v / 5, rv);
            }
            from += __popc(b);
        }
        base += width;
    } while (base < total);
}

// Left and right states of one variable at the face between f[2] and f[3]
// (MDCD_HYBRID: the linear ones).
template <typename T, int INTERP, int RS>
__device__ __forceinline__ void march_pair(const MarchArgs<T> &m, const T *f, T &l, T &r) {
    if constexpr (INTERP == I_WENO5) {
        if constexpr (LaneOf<T>::N == 2) weno5_pair<T>(PairOps(), f[0], f[1], f[2], f[3], f[4], f[5], l, r);
        else weno5_pair<T>(ScalarOps<T>(), f[0], f[1], f[2], f[3], f[4], f[5], l, r);
    } else if constexpr (LaneOf<T>::N == 2) {
        // the order of the one-line form where the Riemann solver runs per line
        constexpr bool ONE = RS != R_HLLC;
        l = mdcd_linear2<ONE>(m.lin, f[0], f[1], f[2], f[3], f[4], f[5]);
        r = mdcd_linear2<ONE>(m.lin, f[5], f[4], f[3], f[2], f[1], f[0]);
    } else {
        l = mdcd_linear(m.lin, f[0], f[1], f[2], f[3], f[4], f[5]);
        r = mdcd_linear(m.lin, f[5], f[4], f[3], f[2], f[1], f[0]);
    }
}

// Every variable of the face between u[2] and u[3]; doubt: march_doubt of the
// two cells (MDCD_HYBRID).
template <typename T, int INTERP, int RS>
__device__ __forceinline__ void march_states(const MarchArgs<T> &m, const T (*u)[5], unsigned doubt, T *UL, T *UR) {
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        const T f[6] = {u[0][q], u[1][q], u[2][q], u[3][q], u[4][q], u[5][q]};
        march_pair<T, INTERP, RS>(m, f, UL[q], UR[q]);
    }
    if constexpr (INTERP == I_MDCD_HYBRID) {
        if (__any_sync(0xffffffffu, doubt != 0)) march_weno<T>(m, u, doubt, UL, UR);
    }
}

template <int DIR, typename T, int INTERP, int RS>
__device__ __forceinline__ void march_flux(const SchemeParams<typename LaneOf<T>::R> &sp, const T *UL, const T *UR, T *F) {
    constexpr bool FORMER = sizeof(typename LaneOf<T>::R) == 4 && INTERP == I_MDCD_HYBRID;
    if constexpr (LaneOf<T>::N == 2) {
        if constexpr (RS == R_HLLC) {
            hllc_flux2<DIR>(UL, UR, sp.gamma, F);
        } else {
            float l[5], r[5], fa[5], fb[5];
#pragma unroll
            for (int q = 0; q < 5; ++q) { l[q] = UL[q].x; r[q] = UR[q].x; }
            riemann<DIR, float, RS, FORMER>(sp, l, r, fa);
#pragma unroll
            for (int q = 0; q < 5; ++q) { l[q] = UL[q].y; r[q] = UR[q].y; }
            riemann<DIR, float, RS, FORMER>(sp, l, r, fb);
#pragma unroll
            for (int q = 0; q < 5; ++q) F[q] = make_float2(fa[q], fb[q]);
        }
    } else {
        riemann<DIR, T, RS, FORMER>(sp, UL, UR, F);
    }
}

// ------------------------------------------------------------------ the kernel

// runge_kutta_3's update of the cells of one thread in increment form (see
// FusedStage, mixed path): U_s = U0 + D_s with the FP32 increments D_1 = dt L0
// and D_2 = (D_1 + dt L1) / 4 kept between stages, U_3 = U0 + 2/3 (D_2 + dt
// L2) in FP64.  The new primitives go to the stage's own FP32 buffer.
template <typename T>
__device__ __forceinline__ void march_stage_mixed(const FusedStage &f, double dt, uint32_t cid, uint32_t c64, const T *rq,
                                                  const double *s0, const T *d, double &smax, double &ke, double &kc) {
    constexpr int LN = LaneOf<T>::N;
    const double irg = f.inv_Rgas;
    T Dn[5], Wn[5], Tn;
#pragma unroll
    for (int h = 0; h < LN; ++h) {
        double U[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            const double rr = (double)march_half(rq[q], h), u0 = s0[q * LN + h];
            const double dp = f.stage == 1 ? 0.0 : (double)march_half(d[q], h);
            if (f.stage == 3) {
                // rounded as written: as the former kernels of two lines and of one
                const double d3 = __fma_rn(dt, rr, dp);
                U[q] = LN == 2 ? __fma_rn(2.0 / 3.0, d3, u0) : __dadd_rn(u0, __dmul_rn(2.0 / 3.0, d3));
            } else {
                const float dn = (float)(f.stage == 1 ? dt * rr : 0.25 * (dp + dt * rr));
                march_set(Dn[q], h, dn);
                U[q] = u0 + (double)dn;
            }
        }
        if (U[0] <= 0.0) U[0] = 1e-12;
        double W[5], ir;
        c2p_fast(U, f.gamma, W, ir);
#pragma unroll
        for (int q = 0; q < 5; ++q) march_set(Wn[q], h, (float)W[q]);
        march_set(Tn, h, (float)(W[4] * ir * irg));
        if (f.stage == 3) {
#pragma unroll
            for (int q = 0; q < 5; ++q) f.Uout[q][c64 + h] = U[q];
            smax = fmax(smax, cfl_speed(U, f.gamma));
            const double y = 0.5 * W[0] * (W[1] * W[1] + W[2] * W[2] + W[3] * W[3]) * f.vol - kc;
            const double t = __dadd_rn(ke, y);
            kc = __dsub_rn(__dsub_rn(t, ke), y);
            ke = t;
        }
    }
    if (f.stage != 3) {
#pragma unroll
        for (int q = 0; q < 5; ++q) *reinterpret_cast<T *>(f.D[q] + cid) = Dn[q];
    }
#pragma unroll
    for (int q = 0; q < 5; ++q) *reinterpret_cast<T *>(f.W32out[q] + cid) = Wn[q];
    *reinterpret_cast<T *>(f.T32out + cid) = Tn;
}

// Shared memory of a block, in bytes: rings of seven node viscous fluxes and
// five faces, the next cell, the old right-hand side and (mixed z-sweep) the
// stage increment, one value of type T per thread and slot; the step-start
// state of the fused stage in FP64; stage 3's sums; line indexes and the detector.  Twelve
// FP64 warps fill an SM's 227 KB.
template <int DIR, typename T>
struct MarchSmem {
    static constexpr bool F64 = sizeof(typename LaneOf<T>::R) == 8;
    static constexpr unsigned slot = MARCH_NT * sizeof(T);
    static constexpr unsigned V = 0, FL = V + 28 * slot, W = FL + 25 * slot, RO = W + 5 * slot, D = RO + 5 * slot;
    static constexpr unsigned ST = D + (DIR == 2 && !F64 ? 5 * slot : 0);
    static constexpr unsigned st_slot = MARCH_NT * sizeof(double) * LaneOf<T>::N;
    static constexpr unsigned ACC = ST + (DIR == 2 ? 5 * st_slot : 0);
    static constexpr unsigned IDX = ACC + (DIR == 2 ? 3 * MARCH_NT * sizeof(double) : 0);
    static constexpr unsigned bytes = IDX + 3 * MARCH_NT * sizeof(uint32_t);
};

// Offset o (o < 2 ring) in a ring of `ring` bytes.
__device__ __forceinline__ unsigned march_ring(unsigned o, unsigned ring) { return min(o, o - ring); }

// Resident blocks asked of the register allocator: twelve warps with 168
// registers (FP64: 0.72 against 0.79 ms along y at 256^3 with eight warps).
// The loop body (some 800 instructions) just fits the instruction cache:
// unrolling it by two, which would save the moves that slide the stencil,
// stalls on instruction fetches (0.76 ms), by three 0.91 ms.
constexpr int MARCH_MINB = 6;
template <int DIR, typename T>
constexpr int march_resident() {
    return DIR == 2 && sizeof(typename LaneOf<T>::R) == 4 && LaneOf<T>::N == 2 ? MARCH_MINB - 1 : MARCH_MINB;
}

template <int DIR, typename T, int INTERP, int RS>
__global__ void __launch_bounds__(MARCH_NT, march_resident<DIR, T>()) march_kernel(const __grid_constant__ MarchArgs<T> m) {
    using R = typename LaneOf<T>::R;
    using S = MarchSmem<DIR, T>;
    constexpr int NT = MARCH_NT, LN = LaneOf<T>::N;
    constexpr bool F64 = sizeof(R) == 8;
    const SweepArgs<R> &a = m.a;
    if (a.done && *a.done) return;  // uniform over the grid
    extern __shared__ __align__(16) unsigned char smem_raw[];
    unsigned char *const mine = smem_raw + threadIdx.x * sizeof(T);
    auto at = [&](unsigned off) -> T * { return reinterpret_cast<T *>(mine + off); };  // off: the same for every thread
    auto slot = [&](unsigned base, int k) -> T * { return at(base + k * S::slot); };
    auto state = [&](int q) -> double * {
        return reinterpret_cast<double *>(smem_raw + S::ST + q * S::st_slot) + threadIdx.x * LN;
    };
    // what the loop needs once per cell stays in shared memory, so that the
    // registers hold the stencil without spilling (a spill goes through the
    // little L1 that the slots leave and stalls on L2)
    volatile double *const acc = reinterpret_cast<volatile double *>(smem_raw + S::ACC) + threadIdx.x;
    volatile uint32_t *const sidx = reinterpret_cast<volatile uint32_t *>(smem_raw + S::IDX) + threadIdx.x;
    const Layout &L = a.L;
    const int n = DIR == 1 ? L.ny : L.nz;
    const bool active = (int)(blockIdx.x * NT + threadIdx.x) < m.nlines;
    const bool per = a.periodic != 0, visc = a.visc != 0, rmw = a.first == 0;
    const int first = DIR == 2 ? a.zlo : 0, last = DIR == 2 ? a.zhi : n;
    const int cs = NG + first + blockIdx.y * m.seg_len, ce = min(cs + m.seg_len, NG + last);  // cells updated
    // 32-bit element indexes: an array of 2^32 elements does not fit the device thirty times over
    const uint32_t lstride = DIR == 1 ? (uint32_t)L.px : (uint32_t)L.px * L.sy;
    const uint32_t vstride = DIR == 1 ? (uint32_t)L.nx : (uint32_t)L.nx * L.ny;
    {
        const int line = min((int)(blockIdx.x * NT + threadIdx.x), m.nlines - 1);  // the last line again where there is none
        const int nxu = L.nx / LN;
        const int other = line / nxu, ix = (line - other * nxu) * LN;
        if (DIR == 1) {
            sidx[0] = (uint32_t)L.at(ix + NG, 0, other + a.zlo + NG);
            sidx[NT] = (uint32_t)(other + a.zlo) * L.ny * L.nx + ix;
        } else {
            sidx[0] = (uint32_t)L.at(ix + NG, other + NG, 0);
            sidx[NT] = (uint32_t)other * L.nx + ix;
            // stage 3: largest wave speed, kinetic energy (compensated sum)
            acc[0] = 0.0; acc[NT] = 0.0; acc[2 * NT] = 0.0;
        }
    }

    auto wrap = [&](int c) { return per ? (c < NG ? c + n : (c >= n + NG ? c - n : c)) : c; };
    auto cell_ok = [&](int c) { return per || (c >= 0 && c < n + 2 * NG); };
    auto fetch_cell = [&](int c) {
        if (cell_ok(c)) {
            const uint32_t id = sidx[0] + (uint32_t)wrap(c) * lstride;
#pragma unroll
            for (int q = 0; q < 5; ++q) march_cp(slot(S::W, q), a.W[q] + id);
        }
    };
    auto fetch_node = [&](int c, unsigned where) {
        if (visc && (per || (c >= NG && c < n + NG))) {
            const uint32_t id = sidx[NT] + (uint32_t)(wrap(c) - NG) * vstride;
#pragma unroll
            for (int q = 0; q < 4; ++q) march_cp(at(S::V + where + q * S::slot), a.V[q] + id);
        }
    };
    // the old right-hand side and the step-start state of cell c
    auto fetch_old = [&](int c) {
        const uint32_t id = sidx[0] + (uint32_t)c * lstride;
        if (rmw) {
#pragma unroll
            for (int q = 0; q < 5; ++q) march_cp(slot(S::RO, q), a.Rhs[q] + id);
        }
        if constexpr (DIR == 2 && F64) {
            if (a.fs.stage > 1) {
#pragma unroll
                for (int q = 0; q < 5; ++q) cp_async(state(q), a.fs.W0[q] + id);
            }
        }
        if constexpr (DIR == 2 && !F64) {
            if (a.fs.stage) {
                const uint32_t id64 = id + (uint32_t)(a.fs.L64.off - L.off);  // the two layouts share the pitch
#pragma unroll
                for (int q = 0; q < 5; ++q) {
                    if constexpr (LN == 2) cp_async16(reinterpret_cast<double2 *>(state(q)), a.fs.U0[q] + id64);
                    else cp_async(state(q), a.fs.U0[q] + id64);
                }
                if (a.fs.stage > 1) {
#pragma unroll
                    for (int q = 0; q < 5; ++q) march_cp(slot(S::D, q), a.fs.D[q] + id);
                }
            }
        }
    };

    // faces f (between cells f and f + 1) the segment differences; the loop
    // starts one before them, for the detector of the first face's own cell
    const int f0 = cs - 3, f1 = ce + 1, fs = f0 - 1;
    constexpr unsigned VR = 28 * S::slot, VS = 4 * S::slot, FR = 25 * S::slot, FS = 5 * S::slot;
    unsigned vo = 0;  // node ring: the slot of node f - 5 (= cu - 3)
    unsigned fo = 0;  // face ring: the slot of face f - 5
    T u[6][5];
    fetch_cell(fs + 3);
    fetch_node(fs + 1, march_ring(vo + 6 * VS, VR));  // node cs - 3; the loop fetches the rest
    cp_async_commit();
    {
        // cells fs - 2 .. fs + 2 into u[1 .. 5]
        T raw[5][5];
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            const int c = fs - 2 + k;
#pragma unroll
            for (int q = 0; q < 5; ++q) raw[k][q] = march_const<T>(1.0);
            if (cell_ok(c)) {
                const uint32_t id = sidx[0] + (uint32_t)wrap(c) * lstride;
#pragma unroll
                for (int q = 0; q < 5; ++q) raw[k][q] = march_ld<T>(a.W[q] + id);
            }
        }
#pragma unroll
        for (int k = 0; k < 6; ++k)
#pragma unroll
            for (int q = 0; q < 5; ++q) u[k][q] = march_const<T>(1.0);
#pragma unroll 1
        for (int k = 0; k < 5; ++k) {  // one copy of the conversion
#pragma unroll
            for (int j = 0; j < 5; ++j)
#pragma unroll
                for (int q = 0; q < 5; ++q) u[j][q] = u[j + 1][q];
            march_cons(a.sp.gamma, raw[0], u[5]);
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int q = 0; q < 5; ++q) raw[j][q] = raw[j + 1][q];
        }
    }
#pragma unroll
    for (int k = 0; k < 25; ++k) *slot(S::FL, k) = march_const<T>(0.0);
    cp_async_commit();
    sidx[2 * NT] = 0;  // march_doubt of cell f
#pragma unroll 1
    for (int f = fs; f <= f1; ++f) {
        // slide the stencil: cells f - 2 .. f + 3 in u[0 .. 5]
#pragma unroll
        for (int k = 0; k < 5; ++k)
#pragma unroll
            for (int q = 0; q < 5; ++q) u[k][q] = u[k + 1][q];
        cp_async_wait<1>();  // cell f + 3
        {
            T w[5];
#pragma unroll
            for (int q = 0; q < 5; ++q) w[q] = *slot(S::W, q);
            if (cell_ok(f + 3)) march_cons(a.sp.gamma, w, u[5]);
        }
        if (f < f1) fetch_cell(f + 4);
        cp_async_commit();
        T fn[5];  // flux of face f
        unsigned doubt = 0;
        if constexpr (INTERP == I_MDCD_HYBRID) {
            const unsigned next = march_doubt<T>(u + 1);
            doubt = sidx[2 * NT] | next;
            sidx[2 * NT] = next;
        }
        if (f >= f0 && (per || (f >= NG - 1 && f < n + NG))) {
            T UL[5], UR[5];
            march_states<T, INTERP, RS>(m, u, doubt, UL, UR);
            march_flux<DIR, T, INTERP, RS>(a.sp, UL, UR, fn);
            if (!per && f == NG - 1 && a.outflow_lo) {  // ghost faces copy the boundary face
#pragma unroll
                for (int q = 0; q < 5; ++q) {
                    *at(S::FL + march_ring(fo + 3 * FS, FR) + q * S::slot) = fn[q];
                    *at(S::FL + march_ring(fo + 4 * FS, FR) + q * S::slot) = fn[q];
                }
            }
        } else if (f >= n + NG && a.outflow_hi) {  // ghost face: a copy of the boundary face, else zero
#pragma unroll
            for (int q = 0; q < 5; ++q) fn[q] = *at(S::FL + march_ring(fo + 4 * FS, FR) + q * S::slot);
        } else {
#pragma unroll
            for (int q = 0; q < 5; ++q) fn[q] = march_const<T>(0.0);
        }
        const int cu = f - 2;  // the cell whose six faces are complete
        cp_async_wait<1>();    // its old right-hand side and step-start state, node f + 1
        if (cu >= cs) {
            const uint32_t cid = sidx[0] + (uint32_t)cu * lstride;
            T rq[5];
            {
                const unsigned o1 = march_ring(fo + FS, FR), o2 = march_ring(fo + 2 * FS, FR),
                               o3 = march_ring(fo + 3 * FS, FR), o4 = march_ring(fo + 4 * FS, FR);
#pragma unroll
                for (int q = 0; q < 5; ++q) {
                    auto F = [&](unsigned o) { return *at(S::FL + o + q * S::slot); };
                    const T ro = rmw ? *slot(S::RO, q) : march_const<T>(0.0);
                    // faces cu - 1/2 and cu + 1/2 are f - 3 and f - 2
                    rq[q] = face_diff(m.dc, m.inv_h, F(o2), F(o3), F(o1), F(o4), F(fo), fn[q], ro);
                }
            }
            const bool edge = !per && (cu - NG < 3 || cu - NG >= n - 3);
            if (visc && !edge) {
                const unsigned v1 = march_ring(vo + VS, VR), v2 = march_ring(vo + 2 * VS, VR), v4 = march_ring(vo + 4 * VS, VR),
                               v5 = march_ring(vo + 5 * VS, VR), v6 = march_ring(vo + 6 * VS, VR);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    auto v = [&](unsigned o) { return *at(S::V + o + q * S::slot); };
                    rq[q + 1] = node_diff(m.vc, m.inv_60h, v(v4), v(v2), v(v5), v(v1), v(v6), v(vo), rq[q + 1]);
                }
            } else if (visc) {
#pragma unroll 1
                for (int q = 0; q < 4; ++q) {
                    auto v = [&](int o) { return *at(S::V + march_ring(vo + (o + 3) * VS, VR) + q * S::slot); };
                    *slot(S::RO, 1 + q) = march_visc_edge(T{}, v, visc_order(cu - NG, n, false), a.dinv);
                }
#pragma unroll
                for (int q = 1; q < 5; ++q) rq[q] = march_add(rq[q], *slot(S::RO, q));
            }
            bool store = active;
            if constexpr (DIR == 2) {
                if (a.fs.stage) {
                    if (active) {
                        const double fdt = a.fs.dt_dev ? *a.fs.dt_dev : a.fs.dt;
                        double smax = 0.0, ke = 0.0, kc = 0.0;
                        if (a.fs.stage == 3) { smax = acc[0]; ke = acc[NT]; kc = acc[2 * NT]; }
                        if constexpr (F64) {
                            double w0[5];
#pragma unroll
                            for (int q = 0; q < 5; ++q) w0[q] = a.fs.stage > 1 ? *state(q) : 0.0;
                            fused_stage_cell(a.fs, fdt, cid, rq, u[0], w0, smax, ke, kc);
                        } else {
                            T d[5];
                            double s0[5 * LN];
#pragma unroll
                            for (int q = 0; q < 5; ++q) {
                                d[q] = a.fs.stage > 1 ? *slot(S::D, q) : march_const<T>(0.0);
#pragma unroll
                                for (int h = 0; h < LN; ++h) s0[q * LN + h] = state(q)[h];
                            }
                            march_stage_mixed<T>(a.fs, fdt, cid, cid + (uint32_t)(a.fs.L64.off - L.off), rq, s0, d, smax, ke, kc);
                        }
                        if (a.fs.stage == 3) { acc[0] = smax; acc[NT] = ke; acc[2 * NT] = kc; }
                    }
                    store = active && a.fs.keep_rhs != 0;
                }
            }
            if (store) {
#pragma unroll
                for (int q = 0; q < 5; ++q) *reinterpret_cast<T *>(a.Rhs[q] + cid) = rq[q];
            }
        }
        // node f + 2 into the slot of node f - 5, face f into that of face f - 5
        if (f < f1 && cu + 1 >= cs) fetch_old(cu + 1);
        if (f < f1) fetch_node(f + 2, vo);
        cp_async_commit();
#pragma unroll
        for (int q = 0; q < 5; ++q) *at(S::FL + fo + q * S::slot) = fn[q];
        fo = march_ring(fo + FS, FR);
        vo = march_ring(vo + VS, VR);
    }
    if constexpr (DIR == 2) {
        if (a.fs.stage == 3)  // uniform: every thread of the block arrives
            block_speed_sum_n<NT>(acc[0], acc[NT] - acc[2 * NT], a.fs.dx,
                                  a.fs.cfl_part + (long)blockIdx.y * gridDim.x + blockIdx.x,
                                  a.fs.ke_part + (long)blockIdx.y * gridDim.x + blockIdx.x);
    }
}

// Cells per segment: the split of the lines that takes least time when a
// resident warp costs `c` per face while the chip is full and a lone warp
// `latency` (in units of c), and every segment computes five faces more.
inline int march_segment(long nblocks, int n, int resident) {
    const int sms = CHIP_SMS;
    const double latency = 12.0;
    int best = n;
    double least = 1e300;
    for (int nseg = 1; nseg <= n; ++nseg) {
        const int len = (n + nseg - 1) / nseg;
        if (nseg > 1 && (n + nseg - 2) / (nseg - 1) == len) continue;
        const long per_sm = (nblocks * ((n + len - 1) / len) + sms - 1) / sms;
        const long full = per_sm / resident, rest = per_sm % resident;
        const double w = MARCH_NT / 32;
        auto pass = [&](double blocks) { return blocks <= 0 ? 0.0 : (blocks * w > latency ? blocks * w : latency); };
        const double t = (full * pass(resident) + pass((double)rest)) * (len + 5 + 3);
        if (t < least * 0.999) { least = t; best = len; }
    }
    return best;
}

template <int DIR, typename T>
inline dim3 march_grid(const SweepArgs<typename LaneOf<T>::R> &a, MarchArgs<T> &m) {
    const int n = DIR == 2 ? a.zhi - a.zlo : a.L.ny;
    m.nlines = a.L.nx / LaneOf<T>::N * (DIR == 2 ? a.L.ny : a.zhi - a.zlo);
    const int nb = (m.nlines + MARCH_NT - 1) / MARCH_NT;
    m.seg_len = march_segment(nb, n, march_resident<DIR, T>());
    return dim3(nb, (n + m.seg_len - 1) / m.seg_len);
}

template <typename T>
inline MarchArgs<T> march_args(const SweepArgs<typename LaneOf<T>::R> &a) {
    MarchArgs<T> m;
    m.a = a;
    using R = typename LaneOf<T>::R;
    auto both = [](R v) {
        if constexpr (LaneOf<T>::N == 2) return make_float2(v, v);
        else return v;
    };
    for (int k = 0; k < 6; ++k) m.lin[k] = both(a.sp.lin[k]);
    for (int k = 0; k < 3; ++k) { m.dc[k] = both(a.dc[k]); m.vc[k] = both(a.vc[k]); }
    m.inv_h = both(a.inv_h);
    m.inv_60h = both(LaneOf<T>::N == 2 ? -a.dinv[2] : a.dinv[2]);
    m.nlines = m.seg_len = 0;
    return m;
}

template <int DIR, typename T, int INTERP, int RS>
inline cudaError_t launch_march(const SweepArgs<typename LaneOf<T>::R> &a, cudaStream_t st) {
    MarchArgs<T> m = march_args<T>(a);
    const dim3 grid = march_grid<DIR, T>(a, m);
    const int smem = (int)MarchSmem<DIR, T>::bytes;
    static unsigned configured = 0;  // one bit per device ordinal
    int dev = 0;
    cudaGetDevice(&dev);
    if (!(configured & (1u << (dev & 31)))) {
        cudaError_t e = cudaFuncSetAttribute(march_kernel<DIR, T, INTERP, RS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             smem);
        if (e != cudaSuccess) return e;
        configured |= 1u << (dev & 31);
    }
    march_kernel<DIR, T, INTERP, RS><<<grid, MARCH_NT, smem, st>>>(m);
    return cudaGetLastError();
}

template <int DIR, typename T>
inline long march_blocks(const SweepArgs<typename LaneOf<T>::R> &a) {
    MarchArgs<T> m;
    const dim3 g = march_grid<DIR, T>(a, m);
    return (long)g.x * g.y;
}
template <int DIR, typename R>
inline long sweep_blocks(const SweepArgs<R> &a) {
    int len;
    const dim3 g = sweep_grid<DIR, R>(a, len);
    return (long)g.x * g.y * g.z;
}

// The scheme's instantiation: the interpolation always compiled in, the
// Riemann solver for the schemes' usual partners.
template <int DIR, typename T>
inline cudaError_t march_select(const SweepArgs<typename LaneOf<T>::R> &a, cudaStream_t st) {
    const auto &sp = a.sp;
    if (sp.interp == I_WENO5)
        return sp.riemann == R_ROE ? launch_march<DIR, T, I_WENO5, R_ROE>(a, st)
                                   : launch_march<DIR, T, I_WENO5, RUNTIME>(a, st);
    if (sp.interp == I_MDCD_LINEAR)
        return sp.riemann == R_HLLC ? launch_march<DIR, T, I_MDCD_LINEAR, R_HLLC>(a, st)
                                    : launch_march<DIR, T, I_MDCD_LINEAR, RUNTIME>(a, st);
    return sp.riemann == R_HLLC ? launch_march<DIR, T, I_MDCD_HYBRID, R_HLLC>(a, st)
                                : launch_march<DIR, T, I_MDCD_HYBRID, RUNTIME>(a, st);
}

}  // namespace ns3d
