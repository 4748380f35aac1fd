// pair.cuh -- the mixed path's FP32 arithmetic on two lines at once.
//
// The sweeps (march.cuh, sweep_line.cuh) carry the same face -- and later the
// same cell -- of two neighbouring lines in the two halves of a float2, so that
//   * the MDCD detector and linear interpolation, the WENO5 pair, the 6th-order
//     half-node difference and the viscous derivative run as sm_100's paired
//     FP32 instructions (add / mul / fma on f32x2: one instruction for both
//     lines),
//   * every shared-memory access moves a 64-bit word (both lines at once), and
//   * along y and z the two lines are x-neighbours, so the global loads,
//     stores and cp.async copies are 8 bytes (16 for the FP64 state).
// HLLC runs paired too (hllc_flux2); the other Riemann solvers and the rare
// WENO branch of the hybrid scheme run per line on the unpacked halves.
//
// Requires an even number of lines across (ny along x, nx along y and z), so a
// pair never straddles the end of the domain and the 8-byte accesses stay
// aligned; other line counts take the same kernels with one line.
#pragma once

#include <cstdlib>
#include <cstring>

#include "sweep.cuh"

namespace ns3d {

__device__ __forceinline__ float2 p2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
// a - b, rounded once (b * -1 is exact)
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }

__device__ __forceinline__ void cp_async8(float2 *smem_dst, const float *gsrc) {
    unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async16(double2 *smem_dst, const double *gsrc) {
    unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gsrc) : "memory");
}

// Paired arithmetic of two lines, for the templates of schemes.cuh
struct PairOps {
    __device__ __forceinline__ float2 c(double x) const { return p2((float)x); }
    __device__ __forceinline__ float2 neg(float2 a) const { return make_float2(-a.x, -a.y); }
    __device__ __forceinline__ float2 add(float2 a, float2 b) const { return add2(a, b); }
    __device__ __forceinline__ float2 sub(float2 a, float2 b) const { return sub2(a, b); }
    __device__ __forceinline__ float2 mul(float2 a, float2 b) const { return mul2(a, b); }
    __device__ __forceinline__ float2 fma(float2 a, float2 b, float2 d) const { return fma2(a, b, d); }
    __device__ __forceinline__ float2 add_quot(float2 g, float2 a, float2 b) const {
        return make_float2(g.x + a.x / b.x, g.y + a.y / b.y);
    }
};

// The scaled sums are taken away from r, not added to it: sub2's multiply-add
// takes a rounded product, where a product and add2 are contracted.  So
// node_diff's scale is minus 1/(60 h) (march_args).
__device__ __forceinline__ float2 face_diff(const float2 *dc, float2 inv_h, float2 l1, float2 r1, float2 l2, float2 r2,
                                            float2 l3, float2 r3, float2 r) {
    float2 t = mul2(sub2(r1, l1), dc[0]);
    t = fma2(sub2(r2, l2), dc[1], t);
    t = fma2(sub2(r3, l3), dc[2], t);
    return sub2(r, mul2(t, inv_h));
}
__device__ __forceinline__ float2 node_diff(const float2 *, float2 minus_inv_60h, float2 p1, float2 m1, float2 q2, float2 m2,
                                            float2 p3, float2 m3, float2 r) {
    float2 t = fma2(p2(-9.f), q2, p3);
    t = fma2(p2(45.f), p1, t);
    t = fma2(p2(-45.f), m1, t);
    t = sub2(fma2(p2(9.f), m2, t), m3);
    return sub2(r, mul2(t, minus_inv_60h));
}

// sum_k c_k f_k (mdcd_linear) for both lines; ONE: the first product rounded
// with the sum and not on its own, as in the one-line form
template <bool ONE>
__device__ __forceinline__ float2 mdcd_linear2(const float2 *c, float2 f0, float2 f1, float2 f2, float2 f3,
                                               float2 f4, float2 f5) {
    float2 s = ONE ? fma2(c[0], f0, mul2(c[1], f1)) : fma2(c[1], f1, mul2(c[0], f0));
    s = fma2(c[2], f2, s);
    s = fma2(c[3], f3, s);
    s = fma2(c[4], f4, s);
    return fma2(c[5], f5, s);
}

// mdcd_smooth for both lines (the detector of interpolation.cpp:135-209 at
// one stencil centre): a and b, the sums of two absolute differences, are
// formed per half (absolute values fold into the scalar adds).
__device__ __forceinline__ void mdcd_smooth2(float2 fm2, float2 fm1, float2 f0, float2 fp1, float2 fp2, bool &sa,
                                             bool &sb) {
    const float eps = float(0.9 * 0.4 / (1.0 - 0.9 * 0.4) * 1e-4);
    const float2 dm = sub2(f0, fm1), tm = add2(fma2(p2(-2.f), fm1, f0), fm2);
    const float2 dp = sub2(f0, fp1), tp = add2(fma2(p2(-2.f), fp1, f0), fp2);
    const float2 A = make_float2(fabsf(dm.x) + fabsf(tm.x), fabsf(dm.y) + fabsf(tm.y));
    const float2 B = make_float2(fabsf(dp.x) + fabsf(tp.x), fabsf(dp.y) + fabsf(tp.y));
    const float2 lhs = fma2(mul2(p2(2.f), A), B, p2(eps));
    const float2 rhs = mul2(p2(0.4f), add2(fma2(A, A, mul2(B, B)), p2(eps)));
    sa = lhs.x > rhs.x;
    sb = lhs.y > rhs.y;
}

// hllc_flux (HLLC_Riemann_solver, InviscousFlux.cpp:449-592) for both lines:
// the side states, wave speeds, S_M and the star flux of the upwind side in
// paired arithmetic; reciprocals, square roots, divisions, minima and the
// side selection per half.  Faces with S_L >= 0 or S_R <= 0 (supersonic,
// rare) and S_M denominators below 1e-12 take the scalar forms per half.
template <int DIR>
__device__ __forceinline__ void hllc_flux2(const float2 *UL, const float2 *UR, float g, float2 *F) {
    const float2 rL = UL[0], rR = UR[0], EL = UL[4], ER = UR[4];
    const float2 irL = make_float2(1.f / rL.x, 1.f / rL.y), irR = make_float2(1.f / rR.x, 1.f / rR.y);
    const float2 uL = mul2(UL[1], irL), vL = mul2(UL[2], irL), wL = mul2(UL[3], irL);
    const float2 uR = mul2(UR[1], irR), vR = mul2(UR[2], irR), wR = mul2(UR[3], irR);
    const float2 gm1 = p2(g - 1.f), mh = p2(-0.5f);
    const float2 pL = mul2(fma2(mul2(mh, rL), fma2(wL, wL, fma2(vL, vL, mul2(uL, uL))), EL), gm1);
    const float2 pR = mul2(fma2(mul2(mh, rR), fma2(wR, wR, fma2(vR, vR, mul2(uR, uR))), ER), gm1);
    const float2 unL = DIR == 0 ? uL : (DIR == 1 ? vL : wL), unR = DIR == 0 ? uR : (DIR == 1 ? vR : wR);
    const float2 tL = mul2(mul2(p2(g), pL), irL), tR = mul2(mul2(p2(g), pR), irR);
    const float2 aL = make_float2(sqrtf(tL.x), sqrtf(tL.y)), aR = make_float2(sqrtf(tR.x), sqrtf(tR.y));
    const float2 dL = sub2(unL, aL), dR = sub2(unR, aR), eL = add2(unL, aL), eR = add2(unR, aR);
    const float2 SL = make_float2(fminf(dL.x, dR.x), fminf(dL.y, dR.y));
    const float2 SR = make_float2(fmaxf(eL.x, eR.x), fmaxf(eL.y, eR.y));
    const float2 cR = sub2(SR, unR), cL = sub2(SL, unL);
    const float2 num = add2(sub2(mul2(mul2(rR, unR), cR), mul2(mul2(rL, unL), cL)), sub2(pL, pR));
    const float2 den = sub2(mul2(rR, cR), mul2(rL, cL));
    float2 SM;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const float n_ = h ? num.y : num.x, d_ = h ? den.y : den.x;
        float sm;
        if (fabsf(d_) > 1e-12f) {
            sm = n_ / d_;
        } else {
            const float sL = sqrtf(h ? rL.y : rL.x), sR = sqrtf(h ? rR.y : rR.x);
            sm = (sL * (h ? unL.y : unL.x) + sR * (h ? unR.y : unR.x)) / (sL + sR);
        }
        if (h) SM.y = sm; else SM.x = sm;
    }
    // the star state of the upwind side, per half
    const bool lx = SM.x >= 0.f, ly = SM.y >= 0.f;
    auto sel = [&](float2 l, float2 r) { return make_float2(lx ? l.x : r.x, ly ? l.y : r.y); };
    const float2 r = sel(rL, rR), ir = sel(irL, irR), u = sel(uL, uR), v = sel(vL, vR), w = sel(wL, wR);
    const float2 E = sel(EL, ER), p = sel(pL, pR), un = sel(unL, unR), Sk = sel(SL, SR);
    const float2 U1 = sel(UL[1], UR[1]), U2 = sel(UL[2], UR[2]), U3 = sel(UL[3], UR[3]);
    const float2 m = mul2(r, un);
    const float2 zero = p2(0.f);
    const float2 Fs0 = m;
    const float2 Fs1 = fma2(m, u, DIR == 0 ? p : zero);
    const float2 Fs2 = fma2(m, v, DIR == 1 ? p : zero);
    const float2 Fs3 = fma2(m, w, DIR == 2 ? p : zero);
    const float2 Fs4 = mul2(add2(E, p), un);
    const float2 dk = sub2(Sk, un), rdk = mul2(r, dk), dS = sub2(Sk, SM);
    const float2 rs = make_float2(rdk.x / dS.x, rdk.y / dS.y);
    const float2 pr = make_float2(p.x / rdk.x, p.y / rdk.y);
    const float2 Es = fma2(sub2(SM, un), add2(SM, pr), mul2(E, ir));
    const float2 us = DIR == 0 ? SM : u, vs = DIR == 1 ? SM : v, ws = DIR == 2 ? SM : w;
    F[0] = fma2(Sk, sub2(rs, r), Fs0);
    F[1] = fma2(Sk, sub2(mul2(rs, us), U1), Fs1);
    F[2] = fma2(Sk, sub2(mul2(rs, vs), U2), Fs2);
    F[3] = fma2(Sk, sub2(mul2(rs, ws), U3), Fs3);
    F[4] = fma2(Sk, sub2(mul2(rs, Es), E), Fs4);
    // supersonic faces: the physical flux of the upwind state
    if (SL.x >= 0.f || SR.x <= 0.f || SL.y >= 0.f || SR.y <= 0.f) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float sl = h ? SL.y : SL.x, sr = h ? SR.y : SR.x;
            if (sl >= 0.f || sr <= 0.f) {
                const float2 *Us = sl >= 0.f ? UL : UR;
                float Uh[5], Fh[5];
#pragma unroll
                for (int q = 0; q < 5; ++q) Uh[q] = h ? Us[q].y : Us[q].x;
                Side<DIR, float> S;
                S.load(Uh, g);
                S.flux(Fh);
#pragma unroll
                for (int q = 0; q < 5; ++q) {
                    if (h) F[q].y = Fh[q]; else F[q].x = Fh[q];
                }
            }
        }
    }
}

// NS3D_SWEEP32=scalar selects the FP32 sweeps with one line per thread or warp
// (those of odd line counts), for comparison.
inline bool sweep32_scalar_forced() {
    const char *v = std::getenv("NS3D_SWEEP32");
    return v && std::strcmp(v, "scalar") == 0;
}

}  // namespace ns3d
