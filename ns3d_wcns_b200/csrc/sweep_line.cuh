// sweep_line.cuh -- the component-wise sweep with a line per warp: every x-sweep,
// and the y- and z-sweeps of small grids (line_takes).
//
// The work and the chunk-relative buffers of sweep_kernel (sweep.cuh), cut for
// the contiguous direction: a warp owns a line (mixed path: two neighbouring
// lines in the halves of a float2) and everything it keeps in shared memory, so
// its phases meet at __syncwarp instead of block barriers.  A chunk holds 64
// faces, two neighbouring ones per lane: their stencils share five of seven
// cells and come as 16-byte loads, and a lane's two updated cells read the
// faces of its neighbours the same way, which leaves a third of the shared
// loads that one face per lane needs.  The first chunk arrives by asynchronous
// copies with one wait, the later ones a chunk ahead.
//
// The one-face kernel (eight lines to a block, a barrier after each phase)
// waited on shared memory and barriers for 3.3 of every 8.3 stall cycles;
// 256^3, one launch along x: FP64 MDCD_HYBRID + HLLC 0.842 -> 0.675 ms, WENO5 +
// Roe 1.083 -> 0.775; FP32 pairs 0.461 -> 0.402 and 0.521 -> 0.487 (0.713,
// 0.789, 0.434, 0.508 with the first chunk loaded position by position).  What
// bounds it now is FP64 issue and latency at twelve warps per SM (192^3, FP64:
// issue slots 51 % and the FP64 pipe 41 % busy, 2.3 TB/s).
#pragma once

#include "march.cuh"

namespace ns3d {

constexpr int XL_WARPS = 4;  // warps (independent lines) per block

// Resident blocks asked of the register allocator: three (168 registers), or
// four (128) where that spills nothing, WENO5 + Roe in FP64 and the one-line FP32
// kernel.  256^3: MDCD_HYBRID + HLLC FP64 0.713 ms with three, 0.846 with four
// (112 bytes spilled), 0.935 with two; WENO5 + Roe FP64 0.834 / 0.794 / 1.04;
// FP32 pairs 0.434 / 0.441 / 0.560; 63^3 FP32 lines 0.027 / 0.023 / 0.027.
template <int DIR, typename T, int INTERP, int RS>
constexpr int xline_resident() {
    if (DIR == 2) return sizeof(typename LaneOf<T>::R) == 4 && LaneOf<T>::N == 2 ? 2 : 3;
    return DIR == 1 ? 3 : sizeof(T) == 4 || (sizeof(typename LaneOf<T>::R) == 8 && INTERP == I_WENO5 && RS == R_ROE) ? 4 : 3;
}

template <int DIR, typename T>
struct XLine {
    static constexpr bool F64 = sizeof(typename LaneOf<T>::R) == 8;
    static constexpr int C = 64;             // faces per chunk, two per lane
    static constexpr int NU = 72, NF = 72, NV = 72;
    //  cells  position p <-> cell fc - 2 + p
    //  faces  position p <-> face fc - 6 + p (a lane's own two start at an even position)
    //  nodes  position p <-> cell fc - 5 + p
    static constexpr int U = 0, F = U + 5 * NU, V = F + 5 * NF, STG = V + 4 * NV, WF = STG + 9 * C;
    //  y, z: the old right-hand side of cells fc - 2 ..; z: their step-start
    //  state in FP64 and (mixed) the stage increment, sums of a lane
    static constexpr int RO = WF + 5 * 6, D = RO + (DIR ? 5 * C : 0), N = D + (DIR == 2 && !F64 ? 5 * C : 0);
    static constexpr int st_off = (N * (int)sizeof(T) + 15) / 16 * 16;
    static constexpr int st_n = DIR == 2 ? 5 * C * LaneOf<T>::N : 0;
    static constexpr int warp_bytes = st_off + (st_n + (DIR == 2 ? 3 * 32 : 0)) * (int)sizeof(double);
    static constexpr int bytes = XL_WARPS * warp_bytes;
    struct alignas(2 * sizeof(T)) Two { T a, b; };
};

// Deals the (lane, face, variable, line) whose detector is in doubt out over
// pairs of the warp's lanes, as march_weno; the stencils are in shared memory.
// doubt: bit q + 5 line (+ NV for the lane's second face).
template <typename T, typename A>
__device__ __forceinline__ void xline_weno(const A &hd, const T *sU, unsigned doubt, T (*UL)[5], T (*UR)[5]) {
    using R = typename LaneOf<T>::R;
    constexpr int LN = LaneOf<T>::N, NV = 5 * LN;
    const int lane = threadIdx.x & 31;
    int total = 0;
#pragma unroll 1
    for (int v = 0; v < 2 * NV; ++v) total += __popc(__ballot_sync(0xffffffffu, (doubt >> v) & 1u));
    int base = 0;
#pragma unroll 1
    do {
        const bool both = total - base > 16;
        const int sh = both ? 0 : 1, width = 32 >> sh;
        int var = 0, nth = 0, off = base + (lane >> sh);  // this lane's task
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
        const R *st = reinterpret_cast<const R *>(sU + q * XLine<0, T>::NU + 2 * src + second) + line;
        R g[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) g[k] = st[k * LN];
        bool keep;
        R sa, sb;
        march_sides(hd, both, (lane & 1) != 0, g, sa, sb, keep);
        if (!both) sb = sa;
        int from = -base;
#pragma unroll
        for (int v = 0; v < 2 * NV; ++v) {
            const unsigned b = __ballot_sync(0xffffffffu, (doubt >> v) & 1u);
            if (!b) continue;
            const int t = from + __popc(b & ((1u << lane) - 1u));
            const int at = (t << sh) & 31;
            const R lv = __shfl_sync(0xffffffffu, sa, at), rv = __shfl_sync(0xffffffffu, sb, at + sh);
            const bool kv = __shfl_sync(0xffffffffu, (int)keep, at);
            if (((doubt >> v) & 1u) && t >= 0 && t < width && !kv) {
                march_set(UL[v / NV][v % NV % 5], v % NV / 5, lv);
                march_set(UR[v / NV][v % NV % 5], v % NV / 5, rv);
            }
            from += __popc(b);
        }
        base += width;
    } while (base < total);
}

template <int DIR, typename T, int INTERP, int RS>
__global__ void __launch_bounds__(32 * XL_WARPS, xline_resident<DIR, T, INTERP, RS>())
sweep_line_kernel(const __grid_constant__ MarchArgs<T> m) {
    using R = typename LaneOf<T>::R;
    using S = XLine<DIR, T>;
    using Two = typename S::Two;
    constexpr int LN = LaneOf<T>::N, C = S::C;
    const SweepArgs<R> &a = m.a;
    if (a.done && *a.done) return;  // uniform over the grid
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, slot = blockIdx.x * XL_WARPS + (threadIdx.x >> 5);
    if (DIR != 2 && slot >= m.nlines) return;  // whole warps; along x and y nothing waits for another warp
    const int unit = min(slot, m.nlines - 1);
    unsigned char *const mine = smem_raw + (threadIdx.x >> 5) * S::warp_bytes;
    T *const sm = reinterpret_cast<T *>(mine);
    T *const sU = sm + S::U, *const sF = sm + S::F, *const sV = sm + S::V, *const stg = sm + S::STG, *const sWrap = sm + S::WF;
    T *const sRO = sm + S::RO, *const sD = sm + S::D;
    double *const sST = reinterpret_cast<double *>(mine + S::st_off), *const acc = sST + S::st_n + lane;
    const Layout &L = a.L;
    const int n = DIR == 0 ? L.nx : (DIR == 1 ? L.ny : L.nz);
    // element strides along the line; 32-bit indexes: an array of 2^32
    // elements does not fit the device thirty times over
    const uint32_t ls = DIR == 0 ? 1u : (DIR == 1 ? (uint32_t)L.px : (uint32_t)L.px * L.sy);
    const uint32_t vs = DIR == 0 ? 1u : (DIR == 1 ? (uint32_t)L.nx : (uint32_t)L.nx * L.ny);
    uint32_t lbase, vbase;
    if (DIR == 0) {
        const int nyu = L.ny / LN, z = unit / nyu + a.zlo, y = (unit % nyu) * LN;
        lbase = (uint32_t)L.at(0, y + NG, z + NG);  // the pair's second line: + px, + nx
        vbase = ((uint32_t)z * L.ny + y) * L.nx;
    } else {
        const int nxu = L.nx / LN, other = unit / nxu, ix = (unit % nxu) * LN;
        lbase = (uint32_t)(DIR == 1 ? L.at(ix + NG, 0, other + a.zlo + NG) : L.at(ix + NG, other + NG, 0));
        vbase = (uint32_t)(DIR == 1 ? (other + a.zlo) * L.ny : other) * L.nx + ix;
    }
    const bool per = a.periodic != 0, visc = a.visc != 0, rmw = DIR != 0 && a.first == 0;
    // the segment's cells [c0, c1) need the faces c0 - 3 .. c1 + 1
    const int first = DIR == 2 ? a.zlo : 0, last = DIR == 2 ? a.zhi : n;
    const int c0 = NG + first + blockIdx.y * m.seg_len, c1 = slot < m.nlines ? min(c0 + m.seg_len, last + NG) : c0;
    const int fb = per ? c0 - NG : max(c0 - NG, NG - 1);    // first face computed from cells
    const int fe = min(c1 + 2, per ? n + 5 : n + NG);       // one past the last computed face
    const int cell_end = min(c1 + 5, per ? n + 8 : n + 6);  // one past the last cell needed
    const bool whole = gridDim.y == 1 && c1 - c0 == n;  // false for a warp without a line
    // a whole periodic line of up to C cells in one chunk: its faces 0 .. n - 1
    // are all there are, and the positions of cells -2 .. 2 update the cells
    // n - 2 .. n + 2 that they repeat (64^3: x 31.1 -> 26.0 us FP64, 28.6 -> 21.1
    // mixed, y mixed 38.0 -> 29.2; the second chunk held five faces)
    const bool ring = per && whole && n <= C && n + 5 > C;
    auto cell = [&](int cu) { return ring && cu < NG ? cu + n : cu; };  // the cell updated at position cu
    auto update = [&](int cu) { return ring ? cu <= n - 3 : cu >= c0 && cu < c1; };
    auto wrap = [&](int c) { return per ? (c < NG ? c + n : (c >= n + NG ? c - n : c)) : c; };
    auto vis_pos = [&](int c) -> int {  // interior index of a node, -1: never read
        if (c < 0 && !ring) return -1;
        int ci = c - NG;
        if (per) { if (ci < 0) ci += n; else if (ci >= n) ci -= n; return ci < n ? ci : -1; }
        return (ci >= 0 && ci < n) ? ci : -1;
    };
    auto cp = [&](T *dst, const R *src, int second) {
        if constexpr (LN == 2 && DIR == 0) { cp_async(&dst->x, src); cp_async(&dst->y, src + second); }
        else march_cp(dst, src);
    };
    if constexpr (DIR == 2) { acc[0] = 0.0; acc[32] = 0.0; acc[64] = 0.0; }

    // ---- first chunk: one wait for all of it, primitives converted in place
#pragma unroll 1
    for (int p = lane; p < S::NV; p += 32) {
        const int c = fb - 5 + p, ci = visc && c < cell_end ? vis_pos(c) : -1;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (ci >= 0) cp(&sV[q * S::NV + p], a.V[q] + vbase + (uint32_t)ci * vs, L.nx);
            else sV[q * S::NV + p] = march_const<T>(0.0);
        }
        if (p >= 3) {
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                if (c < cell_end) cp(&sU[q * S::NU + p - 3], a.W[q] + lbase + (uint32_t)wrap(c) * ls, L.px);
                else sU[q * S::NU + p - 3] = march_const<T>(1.0);
            }
        }
    }
    cp_async_commit();
    cp_async_wait<0>();
#pragma unroll 1
    for (int p = lane; p < S::NV; p += 32) {  // the positions this lane copied
        if (p >= 3) {
            T w[5], U[5];
#pragma unroll
            for (int q = 0; q < 5; ++q) w[q] = sU[q * S::NU + p - 3];
            march_cons(a.sp.gamma, w, U);
#pragma unroll
            for (int q = 0; q < 5; ++q) sU[q * S::NU + p - 3] = U[q];
        }
    }
    unsigned carry = 0;  // march_doubt of cell fc
#pragma unroll 1
    for (int fc = fb; fc - 2 < c1; fc += C) {
        const bool more = !ring && fc + C - 2 < c1;
        if constexpr (DIR != 0) {  // the old right-hand side and step-start state of the cells updated
#pragma unroll 1
            for (int s = lane; s < C; s += 32) {
                const int cu = fc - 2 + s;
                if (!update(cu)) continue;
                const uint32_t id = lbase + (uint32_t)cell(cu) * ls;
                if (rmw) {
#pragma unroll
                    for (int q = 0; q < 5; ++q) march_cp(&sRO[q * C + s], a.Rhs[q] + id);
                }
                if constexpr (DIR == 2 && S::F64) {
                    if (a.fs.stage > 1) {
#pragma unroll
                        for (int q = 0; q < 5; ++q) cp_async(&sST[q * C + s], a.fs.W0[q] + id);
                    }
                }
                if constexpr (DIR == 2 && !S::F64) {
                    if (a.fs.stage) {
                        const uint32_t id64 = id + (uint32_t)(a.fs.L64.off - L.off);  // the two layouts share the pitch
#pragma unroll
                        for (int q = 0; q < 5; ++q) {
                            double *const d = sST + (q * C + s) * LN;
                            if constexpr (LN == 2) cp_async16(reinterpret_cast<double2 *>(d), a.fs.U0[q] + id64);
                            else cp_async(d, a.fs.U0[q] + id64);
                            if (a.fs.stage > 1) march_cp(&sD[q * C + s], a.fs.D[q] + id);
                        }
                    }
                }
            }
            cp_async_commit();
        }
        // stage the next chunk's new cells (cell and node positions 5 + s, 8 + s)
        if (more) {
#pragma unroll 1
            for (int s = lane; s < C; s += 32) {
                const int cn = fc + C + 3 + s;
                if (cn < cell_end) {
                    const uint32_t id = lbase + (uint32_t)wrap(cn) * ls;
#pragma unroll
                    for (int q = 0; q < 5; ++q) cp(&stg[q * C + s], a.W[q] + id, L.px);
                    const int ci = visc ? vis_pos(cn) : -1;
                    if (ci >= 0) {
#pragma unroll
                        for (int q = 0; q < 4; ++q) cp(&stg[(5 + q) * C + s], a.V[q] + vbase + (uint32_t)ci * vs, L.nx);
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
                for (int h = 0; h < 2; ++h) march_pair<T, INTERP, RS>(m, v + h, UL[h][q], UR[h][q]);
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
            for (int h = 0; h < 2; ++h) march_flux<DIR, T, INTERP, RS>(a.sp, UL[h], UR[h], fn[h]);
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
        if (ring) {  // faces -5 .. -1 are faces n - 5 .. n - 1
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int k = f + h - n;
                if (k >= -5 && k < 0) {
#pragma unroll
                    for (int q = 0; q < 5; ++q) sF[q * S::NF + k + 6] = fn[h][q];
                }
            }
        }
        if constexpr (DIR != 0) cp_async_wait<1>();
        __syncwarp();  // faces of this chunk complete, its old right-hand sides landed
        // ---- cells cu = f - 2 and cu + 1: faces cu - 3 .. cu + 3 at positions
        //      2 lane + 1 .. 2 lane + 7, nodes cu - 3 .. cu + 4 at 2 lane .. 2 lane + 7
        const int cu = f - 2;
        const bool up0 = update(cu), up1 = update(cu + 1);
        if (up0 || up1) {
            T rq[2][5], ro[2][5];
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                ro[0][q] = ro[1][q] = march_const<T>(0.0);
                if constexpr (DIR != 0) {
                    if (rmw) {
                        const Two t = *reinterpret_cast<const Two *>(sRO + q * C + s0);
                        ro[0][q] = t.a;
                        ro[1][q] = t.b;
                    }
                }
            }
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
                        rq[h][q] = face_diff(m.dc, m.inv_h, v[3 + h], v[4 + h], v[2 + h], v[5 + h], v[1 + h], v[6 + h], ro[h][q]);
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
                            rq[h][q + 1] = node_diff(m.vc, m.inv_60h, v[4 + h], v[2 + h], v[5 + h], v[1 + h], v[6 + h], v[h], rq[h][q + 1]);
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
                        rq[h][q] = face_diff(m.dc, m.inv_h, v[2], v[3], v[1], v[4], v[0], v[5], ro[h][q]);
                    }
                    const int idx = cu + h - NG;
                    if (visc && idx >= 0 && idx < n) {
                        const int o = visc_order(idx, n, false);
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            auto v = [&](int k) { return sV[q * S::NV + s0 + h + 3 + k]; };
                            if (o == 6)  // the lane's other cell is the one near the boundary
                                rq[h][q + 1] = node_diff(m.vc, m.inv_60h, v(1), v(-1), v(2), v(-2), v(3), v(-3), rq[h][q + 1]);
                            else
                                rq[h][q + 1] = march_add(rq[h][q + 1], march_visc_edge(T{}, v, o, a.dinv));
                        }
                    }
                }
            }
            if constexpr (DIR == 2) {  // the stage takes them in turn, one copy of its code
#pragma unroll
                for (int q = 0; q < 5; ++q) {
                    Two t;
                    t.a = rq[0][q];
                    t.b = rq[1][q];
                    *reinterpret_cast<Two *>(sRO + q * C + s0) = t;
                }
            } else {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (!(h ? up1 : up0)) continue;
                    const uint32_t id = lbase + (uint32_t)cell(cu + h) * ls;
#pragma unroll
                    for (int q = 0; q < 5; ++q) {
                        if constexpr (LN == 2 && DIR == 0) {
                            a.Rhs[q][id] = rq[h][q].x;
                            a.Rhs[q][id + L.px] = rq[h][q].y;
                        } else {
                            *reinterpret_cast<T *>(a.Rhs[q] + id) = rq[h][q];
                        }
                    }
                }
            }
        }
        if constexpr (DIR == 2) {
            __syncwarp();  // right-hand sides of this chunk complete
#pragma unroll 1
            for (int s = lane; s < C; s += 32) {
                const int cl = fc - 2 + s;
                if (!update(cl)) continue;
                const uint32_t cid = lbase + (uint32_t)cell(cl) * ls;
                T r5[5];
#pragma unroll
                for (int q = 0; q < 5; ++q) r5[q] = sRO[q * C + s];
                if (a.fs.stage) {
                    const double fdt = a.fs.dt_dev ? *a.fs.dt_dev : a.fs.dt;
                    double smax = acc[0], ke = acc[32], kc = acc[64];
                    if constexpr (S::F64) {
                        double w0[5], Uc[5];
#pragma unroll
                        for (int q = 0; q < 5; ++q) {
                            w0[q] = a.fs.stage > 1 ? sST[q * C + s] : 0.0;
                            Uc[q] = sU[q * S::NU + s];
                        }
                        fused_stage_cell(a.fs, fdt, cid, r5, Uc, w0, smax, ke, kc);
                    } else {
                        T d[5];
                        double st0[5 * LN];
#pragma unroll
                        for (int q = 0; q < 5; ++q) {
                            d[q] = a.fs.stage > 1 ? sD[q * C + s] : march_const<T>(0.0);
#pragma unroll
                            for (int h = 0; h < LN; ++h) st0[q * LN + h] = sST[(q * C + s) * LN + h];
                        }
                        march_stage_mixed<T>(a.fs, fdt, cid, cid + (uint32_t)(a.fs.L64.off - L.off), r5, st0, d, smax, ke, kc);
                    }
                    acc[0] = smax; acc[32] = ke; acc[64] = kc;
                }
                if (!a.fs.stage || a.fs.keep_rhs) {
#pragma unroll
                    for (int q = 0; q < 5; ++q) *reinterpret_cast<T *>(a.Rhs[q] + cid) = r5[q];
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
    if constexpr (DIR == 2) {
        if (a.fs.stage == 3)  // uniform: every thread of the block arrives
            block_speed_sum_n<32 * XL_WARPS>(acc[0], acc[32] - acc[64], a.fs.dx,
                                             a.fs.cfl_part + (long)blockIdx.y * gridDim.x + blockIdx.x,
                                             a.fs.ke_part + (long)blockIdx.y * gridDim.x + blockIdx.x);
    }
}

// Whole periodic lines of up to C cells take one chunk (see the kernel).
template <int DIR, typename T>
inline bool xline_ring(const SweepArgs<typename LaneOf<T>::R> &a) {
    const int n = DIR == 0 ? a.L.nx : (DIR == 1 ? a.L.ny : a.L.nz);
    return a.periodic && n <= XLine<DIR, T>::C && (DIR != 2 || (a.zlo == 0 && a.zhi == n));
}

template <int DIR, typename T>
inline dim3 xline_grid(const SweepArgs<typename LaneOf<T>::R> &a, int resident, MarchArgs<T> &m) {
    const Layout &L = a.L;
    const int n = DIR == 0 ? L.nx : (DIR == 1 ? L.ny : a.zhi - a.zlo);
    m.nlines = DIR == 0 ? L.ny / LaneOf<T>::N * (a.zhi - a.zlo)
                        : L.nx / LaneOf<T>::N * (DIR == 1 ? a.zhi - a.zlo : L.ny);
    const int nb = (m.nlines + XL_WARPS - 1) / XL_WARPS;
    m.seg_len = xline_ring<DIR, T>(a) ? n : sweep_segment(nb, n, XLine<DIR, T>::C, resident);
    return dim3(nb, (n + m.seg_len - 1) / m.seg_len);
}

template <int DIR, typename T, int INTERP, int RS>
inline cudaError_t launch_sweep_line(const SweepArgs<typename LaneOf<T>::R> &a, cudaStream_t st) {
    MarchArgs<T> m = march_args<T>(a);
    const dim3 grid = xline_grid<DIR, T>(a, xline_resident<DIR, T, INTERP, RS>(), m);
    const int smem = XLine<DIR, T>::bytes;
    static unsigned configured = 0;  // one bit per device ordinal
    int dev = 0;
    cudaGetDevice(&dev);
    if (!(configured & (1u << (dev & 31)))) {
        cudaError_t e = cudaFuncSetAttribute(sweep_line_kernel<DIR, T, INTERP, RS>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        configured |= 1u << (dev & 31);
    }
    sweep_line_kernel<DIR, T, INTERP, RS><<<grid, 32 * XL_WARPS, smem, st>>>(m);
    return cudaGetLastError();
}

template <int DIR, typename T>
inline long xline_blocks(const SweepArgs<typename LaneOf<T>::R> &a) {
    MarchArgs<T> m;
    const dim3 g = xline_grid<DIR, T>(a, xline_resident<DIR, T, I_MDCD_HYBRID, RUNTIME>(), m);
    return (long)g.x * g.y;
}

template <int DIR, typename T>
inline cudaError_t sweep_line_select(const SweepArgs<typename LaneOf<T>::R> &a, cudaStream_t st) {
    const auto &sp = a.sp;
    if (sp.interp == I_WENO5)
        return sp.riemann == R_ROE ? launch_sweep_line<DIR, T, I_WENO5, R_ROE>(a, st)
                                   : launch_sweep_line<DIR, T, I_WENO5, RUNTIME>(a, st);
    if (sp.interp == I_MDCD_LINEAR)
        return sp.riemann == R_HLLC ? launch_sweep_line<DIR, T, I_MDCD_LINEAR, R_HLLC>(a, st)
                                    : launch_sweep_line<DIR, T, I_MDCD_LINEAR, RUNTIME>(a, st);
    return sp.riemann == R_HLLC ? launch_sweep_line<DIR, T, I_MDCD_HYBRID, R_HLLC>(a, st)
                                : launch_sweep_line<DIR, T, I_MDCD_HYBRID, RUNTIME>(a, st);
}

// Along y and z a line's accesses are strided (a block's four warps are
// x-neighbours, so together they use a 32-byte sector), and the marching kernel
// with its coalesced lanes is three times as fast on a full chip.  But it has a
// thread per line and walks it a face at a time: on a small grid it is latency,
// or cuts the lines into segments that recompute five faces each.  The line
// kernel takes the grids whose chunks of 64 faces fit the chip's resident warps
// at most twice along y and once along z, where the fused stage adds more
// strided traffic.  us, march / line: FP64 y 16x16x16 14.7 / 10.5, 32^3 18.9 /
// 12.8, 42 x 28 x 42 35.2 / 16.7, 56 x 59 x 56 (3136 chunks) 45.9 / 32.3, 48 x
// 120 x 48 (4608) 45.0 / 58.1, 64^3 (4096) WENO5 + Roe 35.4 / 35.3, MDCD_LINEAR
// 23.1 / 35.7; z 32^3 20.0 / 16.0, 42^3 (1764) 34.2 / 24.6, 48^3 (2304) WENO5 +
// Roe 28.9 / 28.5, 56^3 (3136) 35.4 / 43.5; FP32 pairs y 48^3 31.4 / 18.7, 56 x
// 120 x 56 (3136) 39.6 / 35.5; z 48^3 (1152) 31.3 / 23.5, 59 x 48 x 48 (1416)
// 33.8 / 36.1.
template <int DIR, typename T>
inline bool line_takes(const SweepArgs<typename LaneOf<T>::R> &a) {
    const int n = DIR == 1 ? a.L.ny : a.zhi - a.zlo, C = XLine<DIR, T>::C;
    const long lines = (long)(a.L.nx / LaneOf<T>::N) * (DIR == 1 ? a.zhi - a.zlo : a.L.ny);
    const long warps = (long)CHIP_SMS * XL_WARPS * xline_resident<DIR, T, I_MDCD_HYBRID, RUNTIME>();
    return lines * (xline_ring<DIR, T>(a) ? 1 : (n + 5 + C - 1) / C) <= (DIR == 1 ? 2 : 1) * warps;
}
template <int DIR, typename T>
inline cudaError_t line_or_march(const SweepArgs<typename LaneOf<T>::R> &a, cudaStream_t st) {
    return line_takes<DIR, T>(a) ? sweep_line_select<DIR, T>(a, st) : march_select<DIR, T>(a, st);
}
template <int DIR, typename T>
inline long line_or_march_blocks(const SweepArgs<typename LaneOf<T>::R> &a) {
    return line_takes<DIR, T>(a) ? xline_blocks<DIR, T>(a) : march_blocks<DIR, T>(a);
}

}  // namespace ns3d
