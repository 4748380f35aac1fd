// sweep_line.cuh -- the component-wise sweep along x, one line per warp.
//
// The work and the chunk-relative buffers of sweep_kernel (sweep.cuh), cut for
// the contiguous direction: a warp owns a line (mixed path: two y-neighbouring
// lines in the halves of a float2) and everything it keeps in shared memory, so
// its phases meet at __syncwarp instead of block barriers.  A chunk holds 64
// faces, two neighbouring ones per lane: their stencils share five of seven
// cells and come as 16-byte loads, and a lane's two updated cells read the
// faces of its neighbours the same way, which leaves a third of the shared
// loads that one face per lane needs.  The one-face kernel (eight lines to a
// block, a barrier after each phase) waited on shared memory and barriers for
// 3.3 of every 8.3 stall cycles; 256^3, one launch: FP64 MDCD_HYBRID + HLLC
// 0.842 -> 0.713 ms, WENO5 + Roe 1.083 -> 0.794; FP32 pairs 0.461 -> 0.434 and
// 0.521 -> 0.508.  What bounds it now is FP64 issue and latency at twelve warps
// per SM.
#pragma once

#include "march.cuh"

namespace ns3d {

constexpr int XL_WARPS = 4;  // warps (independent lines) per block

// Resident blocks asked of the register allocator: three (168 registers), or
// four (128) where that spills nothing, WENO5 + Roe in FP64 and the one-line FP32
// kernel.  256^3: MDCD_HYBRID + HLLC FP64 0.713 ms with three, 0.846 with four
// (112 bytes spilled), 0.935 with two; WENO5 + Roe FP64 0.834 / 0.794 / 1.04;
// FP32 pairs 0.434 / 0.441 / 0.560; 63^3 FP32 lines 0.027 / 0.023 / 0.027.
template <typename T, int INTERP, int RS>
constexpr int xline_resident() {
    return sizeof(T) == 4 || (sizeof(typename LaneOf<T>::R) == 8 && INTERP == I_WENO5 && RS == R_ROE) ? 4 : 3;
}

template <typename T>
struct XLine {
    static constexpr int C = 64;             // faces per chunk, two per lane
    static constexpr int NU = 72, NF = 72, NV = 72;
    //  cells  position p <-> cell fc - 2 + p
    //  faces  position p <-> face fc - 6 + p (a lane's own two start at an even position)
    //  nodes  position p <-> cell fc - 5 + p
    static constexpr int U = 0, F = U + 5 * NU, V = F + 5 * NF, ST = V + 4 * NV, WF = ST + 9 * C, N = WF + 5 * 6;
    static constexpr int warp_bytes = N * (int)sizeof(T);
    static constexpr int bytes = XL_WARPS * warp_bytes;
    struct alignas(2 * sizeof(T)) Two { T a, b; };
};

// Deals the (lane, face, variable, line) whose detector is in doubt out over
// the warp's lanes, as march_weno; the stencils are in shared memory.
// doubt: bit q + 5 line (+ NV for the lane's second face).
template <typename T, typename A>
__device__ __forceinline__ void xline_weno(const A &hd, const T *sU, unsigned doubt, T (*UL)[5], T (*UR)[5]) {
    using R = typename LaneOf<T>::R;
    constexpr int LN = LaneOf<T>::N, NV = 5 * LN;
    const int lane = threadIdx.x & 31;
    int total = 0;
#pragma unroll 1
    for (int v = 0; v < 2 * NV; ++v) total += __popc(__ballot_sync(0xffffffffu, (doubt >> v) & 1u));
#pragma unroll 1
    for (int base = 0; base < total; base += 32) {
        int var = 0, nth = 0, off = base + lane;  // this lane's task
        unsigned mask = 0;
#pragma unroll 1
        for (int v = 0; v < 2 * NV; ++v) {
            const unsigned b = __ballot_sync(0xffffffffu, (doubt >> v) & 1u);
            const int c = __popc(b);
            if (off >= 0 && off < c) { var = v; mask = b; nth = off; }
            off -= c;
        }
        const int src = march_nth_bit(mask, nth) & 31, second = var >= NV, vl = var - (second ? NV : 0);
        const int line = vl >= 5, q = vl - 5 * line;
        const R *st = reinterpret_cast<const R *>(sU + q * XLine<T>::NU + 2 * src + second) + line;
        R g[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) g[k] = st[k * LN];
        bool keep = false;  // the linear states stay
        if constexpr (sizeof(R) == 8)
            keep = mdcd_smooth(g[0], g[1], g[2], g[3], g[4]) && mdcd_smooth(g[1], g[2], g[3], g[4], g[5]);
        const R l = mdcd_weno_branch(hd, g[0], g[1], g[2], g[3], g[4], g[5]);
        const R r = mdcd_weno_branch(hd, g[5], g[4], g[3], g[2], g[1], g[0]);
        int from = -base;
#pragma unroll
        for (int v = 0; v < 2 * NV; ++v) {
            const unsigned b = __ballot_sync(0xffffffffu, (doubt >> v) & 1u);
            if (!b) continue;
            const int t = from + __popc(b & ((1u << lane) - 1u));
            const R lv = __shfl_sync(0xffffffffu, l, t & 31), rv = __shfl_sync(0xffffffffu, r, t & 31);
            const bool kv = __shfl_sync(0xffffffffu, (int)keep, t & 31);
            if (((doubt >> v) & 1u) && t >= 0 && t < 32 && !kv) {
                march_set(UL[v / NV][v % NV % 5], v % NV / 5, lv);
                march_set(UR[v / NV][v % NV % 5], v % NV / 5, rv);
            }
            from += __popc(b);
        }
    }
}

template <typename T, int INTERP, int RS>
__global__ void __launch_bounds__(32 * XL_WARPS, xline_resident<T, INTERP, RS>()) sweep_line_kernel(const __grid_constant__ MarchArgs<T> m) {
    using R = typename LaneOf<T>::R;
    using S = XLine<T>;
    using Two = typename S::Two;
    constexpr int LN = LaneOf<T>::N, C = S::C;
    const SweepArgs<R> &a = m.a;
    if (a.done && *a.done) return;  // uniform over the grid
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, unit = blockIdx.x * XL_WARPS + (threadIdx.x >> 5);
    if (unit >= m.nlines) return;  // whole warps; nothing below waits for another warp
    T *const sm = reinterpret_cast<T *>(smem_raw + (threadIdx.x >> 5) * S::warp_bytes);
    T *const sU = sm + S::U, *const sF = sm + S::F, *const sV = sm + S::V, *const stg = sm + S::ST, *const sWrap = sm + S::WF;
    const Layout &L = a.L;
    const int n = L.nx;
    const int nyu = L.ny / LN, z = unit / nyu + a.zlo, y = (unit % nyu) * LN;
    const long lbase = L.at(0, y + NG, z + NG), vbase = ((long)z * L.ny + y) * L.nx;  // the pair's second line: + px, + nx
    const bool per = a.periodic != 0, visc = a.visc != 0;
    // the segment's cells [c0, c1) need the faces c0 - 3 .. c1 + 1
    const int c0 = NG + blockIdx.y * m.seg_len, c1 = min(c0 + m.seg_len, n + NG);
    const int fb = per ? c0 - NG : max(c0 - NG, NG - 1);    // first face computed from cells
    const int fe = min(c1 + 2, per ? n + 5 : n + NG);       // one past the last computed face
    const int cell_end = min(c1 + 5, per ? n + 8 : n + 6);  // one past the last cell needed
    const bool whole = gridDim.y == 1;
    auto wrap = [&](int c) { return per ? (c < NG ? c + n : (c >= n + NG ? c - n : c)) : c; };
    auto vis_pos = [&](int c) -> int {  // interior index of a node, -1: never read
        if (c < 0) return -1;
        int ci = c - NG;
        if (per) { if (ci < 0) ci += n; else if (ci >= n) ci -= n; return ci < n ? ci : -1; }
        return (ci >= 0 && ci < n) ? ci : -1;
    };
    auto ld = [&](const R *p, long second) -> T {
        if constexpr (LN == 2) return make_float2(p[0], p[second]);
        else return p[0];
    };
    auto cp = [&](T *dst, const R *src, long second) {
        if constexpr (LN == 2) { cp_async(&dst->x, src); cp_async(&dst->y, src + second); }
        else cp_async(dst, src);
    };

    // ---- first chunk
    for (int p = lane; p < S::NV; p += 32) {
        const int c = fb - 5 + p, ci = visc ? vis_pos(c) : -1;
#pragma unroll
        for (int q = 0; q < 4; ++q) sV[q * S::NV + p] = ci >= 0 ? ld(a.V[q] + vbase + ci, L.nx) : march_const<T>(0.0);
        if (p >= 3) {
            T w[5], U[5];
#pragma unroll
            for (int q = 0; q < 5; ++q) w[q] = c < cell_end ? ld(a.W[q] + lbase + wrap(c), L.px) : march_const<T>(1.0);
            march_cons(a.sp.gamma, w, U);
#pragma unroll
            for (int q = 0; q < 5; ++q) sU[q * S::NU + p - 3] = U[q];
        }
    }
    unsigned carry = 0;  // march_doubt of cell fc
#pragma unroll 1
    for (int fc = fb; fc - 2 < c1; fc += C) {
        const bool more = fc + C - 2 < c1;
        // stage the next chunk's new cells (cell and node positions 5 + s, 8 + s)
        if (more) {
#pragma unroll 1
            for (int s = lane; s < C; s += 32) {
                const int cn = fc + C + 3 + s;
                if (cn < cell_end) {
                    const long id = lbase + wrap(cn);
#pragma unroll
                    for (int q = 0; q < 5; ++q) cp(&stg[q * C + s], a.W[q] + id, L.px);
                    const int ci = visc ? vis_pos(cn) : -1;
                    if (ci >= 0) {
#pragma unroll
                        for (int q = 0; q < 4; ++q) cp(&stg[(5 + q) * C + s], a.V[q] + vbase + ci, L.nx);
                    }
                }
            }
        }
        cp_async_commit();
        __syncwarp();  // buffers of this chunk complete
        // ---- faces f and f + 1: cell positions 2 lane .. 2 lane + 6
        const int s0 = 2 * lane, f = fc + s0;
        T fn[2][5];
        if (per && whole && fc >= n) {  // only faces n .. n + 4, copies of faces 0 .. 4 (the same wrapped cells)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int q = 0; q < 5; ++q) fn[h][q] = sWrap[q * 6 + min(f + h - n, 5)];
        } else {
            T UL[2][5], UR[2][5];
            unsigned first = 0, d1 = 0, d2 = 0;  // march_doubt of cells f, f + 1, f + 2
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                T v[8];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const Two t = *reinterpret_cast<const Two *>(sU + q * S::NU + s0 + 2 * k);
                    v[2 * k] = t.a;
                    v[2 * k + 1] = t.b;
                }
                if constexpr (INTERP == I_MDCD_HYBRID) {
                    d1 |= march_doubt1(v + 1) << q;
                    d2 |= march_doubt1(v + 2) << q;
                    if (fc == fb && lane == 0) first |= march_doubt1(v) << q;
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) march_pair<T, INTERP>(m, v + h, UL[h][q], UR[h][q]);
            }
            if constexpr (INTERP == I_MDCD_HYBRID) {
                unsigned d0 = __shfl_up_sync(0xffffffffu, d2, 1);
                if (lane == 0) d0 = fc == fb ? first : carry;
                carry = __shfl_sync(0xffffffffu, d2, 31);
                // beyond the last face the buffers hold nothing to decide on
                const unsigned w0 = f < fe ? d0 | d1 : 0u, w1 = f + 1 < fe ? d1 | d2 : 0u, doubt = w0 | w1 << 5 * LN;
                if (__any_sync(0xffffffffu, doubt != 0)) xline_weno<T>(a.sp.hd, sU, doubt, UL, UR);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) march_flux<0, T, RS>(a.sp, UL[h], UR[h], fn[h]);
            if (per && whole && f < 5) {  // first chunk (fb = 0): faces 0 .. 5
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int q = 0; q < 5; ++q) sWrap[q * 6 + f + h] = fn[h][q];
            }
        }
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            Two t;
            t.a = fn[0][q];
            t.b = fn[1][q];
            *reinterpret_cast<Two *>(sF + q * S::NF + s0 + 6) = t;
        }
        __syncwarp();  // faces of this chunk complete
        // ---- cells cu = f - 2 and cu + 1: faces cu - 3 .. cu + 3 at positions
        //      2 lane + 1 .. 2 lane + 7, nodes cu - 3 .. cu + 4 at 2 lane .. 2 lane + 7
        const int cu = f - 2;
        const bool up0 = cu >= c0 && cu < c1, up1 = cu + 1 >= c0 && cu + 1 < c1;
        if (up0 || up1) {
            T rq[2][5];
            const bool edge = !per && (cu - NG < 3 || cu + 1 - NG >= n - 3);
            if (!edge) {
#pragma unroll
                for (int q = 0; q < 5; ++q) {
                    T v[8];
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        const Two t = *reinterpret_cast<const Two *>(sF + q * S::NF + s0 + 2 * k);
                        v[2 * k] = t.a;
                        v[2 * k + 1] = t.b;
                    }
                    v[6] = fn[0][q];
                    v[7] = fn[1][q];
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        rq[h][q] = diff3(m.dc, v[3 + h], v[4 + h], v[2 + h], v[5 + h], v[1 + h], v[6 + h], march_const<T>(0.0));
                }
                if (visc) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        T v[8];
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const Two t = *reinterpret_cast<const Two *>(sV + q * S::NV + s0 + 2 * k);
                            v[2 * k] = t.a;
                            v[2 * k + 1] = t.b;
                        }
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            rq[h][q + 1] = diff3(m.vc, v[4 + h], v[2 + h], v[5 + h], v[1 + h], v[6 + h], v[h], rq[h][q + 1]);
                    }
                }
            } else {
                // within 3 cells of a boundary: ghost faces (Outflow copies, else
                // zero) and reduced viscous orders, a cell and variable at a time
                const int p_lo = (NG - 1) - (fc - 6), p_hi = (n + NG - 1) - (fc - 6);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
#pragma unroll
                    for (int q = 0; q < 5; ++q) {
                        T v[6];
#pragma unroll
                        for (int k = 0; k < 6; ++k) {
                            int p = s0 + 1 + h + k;
                            const int ff = fc - 6 + p;
                            bool zero = false;
                            if (ff < NG - 1) { if (a.outflow_lo) p = p_lo; else zero = true; }
                            else if (ff > n + NG - 1) { if (a.outflow_hi) p = p_hi; else zero = true; }
                            v[k] = zero ? march_const<T>(0.0) : sF[q * S::NF + p];
                        }
                        rq[h][q] = diff3(m.dc, v[2], v[3], v[1], v[4], v[0], v[5], march_const<T>(0.0));
                    }
                    const int idx = cu + h - NG;
                    if (visc && idx >= 0 && idx < n) {
                        const int o = visc_order(idx, n, false);
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const T vd = march_visc_edge(T{}, [&](int k) { return sV[q * S::NV + s0 + h + 3 + k]; }, o, a.dinv);
                            rq[h][q + 1] = march_add(rq[h][q + 1], vd);
                        }
                    }
                }
            }
            // store: the second cell of the lane lies next to the first
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (!(h ? up1 : up0)) continue;
                const long id = lbase + cu + h;
#pragma unroll
                for (int q = 0; q < 5; ++q) {
                    if constexpr (LN == 2) {
                        a.Rhs[q][id] = rq[h][q].x;
                        a.Rhs[q][id + L.px] = rq[h][q].y;
                    } else {
                        a.Rhs[q][id] = rq[h][q];
                    }
                }
            }
        }
        if (!more) break;
        cp_async_wait<0>();
        __syncwarp();  // buffer reads of this chunk done; staged cells landed
        // ---- move the tails to the front, append the staged cells
        {
            T tu[5], tf[5], tv[4];
            if (lane < 8) {
#pragma unroll
                for (int q = 0; q < 5; ++q) {
                    tu[q] = sU[q * S::NU + min(C + lane, S::NU - 1)];
                    tf[q] = sF[q * S::NF + min(C + lane, S::NF - 1)];
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) tv[q] = sV[q * S::NV + C + lane];
            }
            __syncwarp();
            if (lane < 8) {
#pragma unroll
                for (int q = 0; q < 4; ++q) sV[q * S::NV + lane] = tv[q];
#pragma unroll
                for (int q = 0; q < 5; ++q) {
                    if (lane < 5) sU[q * S::NU + lane] = tu[q];
                    if (lane < 6) sF[q * S::NF + lane] = tf[q];
                }
            }
#pragma unroll 1
            for (int s = lane; s < C; s += 32) {
                T w[5], U[5];
                const bool ok = fc + C + 3 + s < cell_end;
#pragma unroll
                for (int q = 0; q < 5; ++q) w[q] = ok ? stg[q * C + s] : march_const<T>(1.0);
                march_cons(a.sp.gamma, w, U);
#pragma unroll
                for (int q = 0; q < 5; ++q) sU[q * S::NU + 5 + s] = U[q];
                if (visc) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) sV[q * S::NV + 8 + s] = ok ? stg[(5 + q) * C + s] : march_const<T>(0.0);
                }
            }
        }
    }
}

template <typename T, int INTERP, int RS>
inline cudaError_t launch_sweep_line(const SweepArgs<typename LaneOf<T>::R> &a, cudaStream_t st) {
    MarchArgs<T> m = march_args<T>(a);
    m.nlines = a.L.ny / LaneOf<T>::N * (a.zhi - a.zlo);
    const int nb = (m.nlines + XL_WARPS - 1) / XL_WARPS;
    m.seg_len = sweep_segment(nb, a.L.nx, XLine<T>::C, xline_resident<T, INTERP, RS>());
    static unsigned configured = 0;  // one bit per device ordinal
    int dev = 0;
    cudaGetDevice(&dev);
    if (!(configured & (1u << (dev & 31)))) {
        cudaError_t e = cudaFuncSetAttribute(sweep_line_kernel<T, INTERP, RS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             XLine<T>::bytes);
        if (e != cudaSuccess) return e;
        configured |= 1u << (dev & 31);
    }
    sweep_line_kernel<T, INTERP, RS><<<dim3(nb, (a.L.nx + m.seg_len - 1) / m.seg_len), 32 * XL_WARPS, XLine<T>::bytes, st>>>(m);
    return cudaGetLastError();
}

template <typename T>
inline cudaError_t sweep_line_select(const SweepArgs<typename LaneOf<T>::R> &a, cudaStream_t st) {
    const auto &sp = a.sp;
    if (sp.interp == I_WENO5)
        return sp.riemann == R_ROE ? launch_sweep_line<T, I_WENO5, R_ROE>(a, st) : launch_sweep_line<T, I_WENO5, RUNTIME>(a, st);
    if (sp.interp == I_MDCD_LINEAR)
        return sp.riemann == R_HLLC ? launch_sweep_line<T, I_MDCD_LINEAR, R_HLLC>(a, st)
                                    : launch_sweep_line<T, I_MDCD_LINEAR, RUNTIME>(a, st);
    return sp.riemann == R_HLLC ? launch_sweep_line<T, I_MDCD_HYBRID, R_HLLC>(a, st)
                                : launch_sweep_line<T, I_MDCD_HYBRID, RUNTIME>(a, st);
}

}  // namespace ns3d
