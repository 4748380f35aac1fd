"""What a program that uses ns3d_wcns_b200 has it do, as measurable cases.

Every case goes through the public Python entry points over the C ABI
(ns3d_wcns_b200.solver.Solver, ns3d_wcns_b200.batch.Batch):

  step        compute_timestep + rk3_step from a host loop (the drop-in's own loop)
  fixed       rk3_steps: fixed-dt steps in one call
  advance     time_advance: the device-resident adaptive loop, then the monitors where a run prints them
  adjoint     adjoint_kinetic_energy: checkpointed forward and backward pass
  vjp         vjp_rk3_step: one reverse step between host arrays
  batch       Batch.run over many shock tubes of uneven length, then every result downloaded

``exact`` is a plain torch FP64 restatement of the scheme (interpolation,
Riemann solver, viscous terms, boundary treatment, SSP-RK3, CFL step), with
reverse mode by torch.autograd.
"""
import math

import numpy as np
import torch

from ns3d_wcns_b200.batch import Batch
from ns3d_wcns_b200.config import GridDesc, make_params
from ns3d_wcns_b200.solver import Solver

WENO5, LINEAR, HYBRID = 0, 2, 3
ROE, RUSANOV, HLLC, HLL = 0, 1, 2, 3
PERIODIC, WALL, SYMMETRY, OUTFLOW = 0, 1, 2, 3
PRIMITIVE, RHS = 0, 2
GAMMA = 1.4
TUBES = (200, 400, 800, 1600)

DEFAULT = {"kind": "advance", "nx": 64, "ny": 64, "nz": 64, "interp": HYBRID, "riemann": HLLC, "char": False,
           "mixed": False, "bc": "000000", "re": 400.0, "flow": "turbulence", "steps": 1, "every": 1, "dt": 1e-3,
           "monitor": False, "tubes": 0}


def case(name=None, **kw):
    c = dict(DEFAULT, **kw)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: a 16^3 box, one right-hand side and one adaptive step from the host loop
        case("step_16", kind="step", nx=16, ny=16, nz=16, interp=WENO5, riemann=ROE, re=100.0, monitor=True),
        # a 32^3 validation run with a fixed time step, ten steps in one call
        case("fixed_32_weno_roe", kind="fixed", nx=32, ny=32, nz=32, interp=WENO5, riemann=ROE, re=100.0, steps=10),
        # decaying turbulence at 64^3 on the device loop, its monitors read every twelve steps
        case("advance_64_monitored", nx=64, ny=64, nz=64, steps=12, monitor=True),
        # the benchmark's grid and scheme: 256^3, MDCD_HYBRID + HLLC, adaptive steps, plain FP64 path
        case("advance_256_fp64", nx=256, ny=256, nz=256, steps=3),
        # a production grid on the mixed FP32/FP64 path
        case("advance_384_mixed", nx=384, ny=384, nz=384, steps=2, mixed=True),
        # a ragged box between walls and an outflow, viscous, WENO5 + Roe, stepped from the host
        case("step_bounded_ragged", kind="step", nx=150, ny=66, nz=91, interp=WENO5, riemann=ROE, bc="331100", re=400.0,
             flow="pulse", steps=2),
        # odd line counts on the mixed path (outflow in x, symmetry in z)
        case("advance_odd_mixed", nx=129, ny=95, nz=77, interp=LINEAR, riemann=HLLC, bc="330022", flow="pulse", steps=3,
             mixed=True),
        # characteristic-wise reconstruction, as runs with shocks choose it
        case("step_characteristic", kind="step", nx=96, ny=64, nz=64, interp=WENO5, riemann=HLL, char=True, bc="330000",
             flow="pulse", steps=2),
        # the solver's default problem: the two-dimensional Riemann problem, inviscid, outflow, a thin box
        case("advance_riemann_2d", nx=384, ny=384, nz=4, interp=WENO5, riemann=HLLC, bc="333300", re=math.inf,
             flow="quadrants", steps=6),
        # gradient of the final kinetic energy with respect to the initial velocity, checkpointed
        case("adjoint_64", kind="adjoint", nx=64, ny=64, nz=64, interp=WENO5, riemann=ROE, re=200.0, steps=8, every=4,
             dt=2e-3),
        # one reverse step of the benchmark scheme between host arrays, uneven sides
        case("vjp_step_ragged", kind="vjp", nx=72, ny=50, nz=45, re=200.0, dt=2e-3),
        # 256 shock tubes of uneven length, 96 steps, results to the host
        case("batch_256_tubes", kind="batch", nx=1600, ny=4, nz=4, interp=WENO5, riemann=ROE, bc="330000", re=math.inf,
             flow="tubes", steps=96, tubes=256),
    ]


def draw(rng):
    side = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(["advance", "advance", "step", "step", "fixed", "adjoint", "vjp", "batch"])
    if kind == "batch":
        n = side(8, 256)
        return case(kind=kind, nx=1600, ny=4, nz=4, interp=WENO5, riemann=ROE, bc="330000", re=math.inf, flow="tubes",
                    steps=24 * rng.randint(1, 4), tubes=n)
    if kind in ("adjoint", "vjp"):
        it, rs = rng.choice([(WENO5, ROE), (LINEAR, HLLC), (HYBRID, HLLC)] if kind == "vjp" else [(WENO5, ROE), (LINEAR, HLLC)])
        steps = rng.randint(2, 8)
        return case(kind=kind, nx=side(16, 80), ny=side(16, 80), nz=side(16, 64), interp=it, riemann=rs, re=200.0,
                    steps=steps, every=rng.randint(1, steps), dt=1e-3)
    bc = rng.choice(["000000", "000000", "331100", "330022", "333300", "110033"])
    it, rs = rng.choice([(WENO5, ROE), (HYBRID, HLLC), (HYBRID, HLLC), (LINEAR, HLLC), (WENO5, HLLC), (WENO5, HLL)])
    per = bc == "000000"
    n = [side(12, 256) for _ in range(3)]
    while n[0] * n[1] * n[2] > 256 ** 3 // 2:
        n[n.index(max(n))] //= 2
    mixed = rng.random() < 0.35
    return case(kind=kind, nx=n[0], ny=n[1], nz=n[2], interp=it if per or it != HYBRID else WENO5, riemann=rs,
                char=not mixed and rng.random() < 0.15, mixed=mixed, bc=bc, re=rng.choice([100.0, 400.0, 400.0, math.inf]),
                flow="turbulence" if per else "pulse", steps=rng.randint(1, 4), dt=2e-4, monitor=not mixed and rng.random() < 0.3)


# ------------------------------------------------------------------- inputs

def lengths(c):
    if c["flow"] == "quadrants":
        return 1.0, 1.0, c["nz"] / c["nx"]
    # a spacing of 2 pi / 64 or finer, near-cubic cells
    h = 2 * math.pi / max(c["nx"], c["ny"], c["nz"], 64)
    return (2 * math.pi,) * 3 if c["nx"] == c["ny"] == c["nz"] else (h * c["nx"], h * c["ny"], h * c["nz"])


def params(c):
    L = lengths(c)
    P, G = make_params(n=(c["nx"], c["ny"], c["nz"]), L=L, gamma=GAMMA, Ma=mach(c), Re=c["re"], Pr=0.72, cfl=0.4,
                       dt_fixed=-1.0 if c["kind"] != "fixed" else c["dt"], interpolation=c["interp"],
                       riemann=c["riemann"], char_recon=c["char"], bcs=tuple(int(x) for x in c["bc"]),
                       precision=int(c["mixed"]))
    return P, G


def mach(c):
    return 1.0 if c["flow"] in ("tubes", "quadrants") else 0.3


def wave_numbers(n):
    return torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device="cuda")


def fields(c, seed):
    """(5, nz, ny, nx) primitives (rho, u, v, w, p) on the GPU, from the seed alone."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    n = (c["nz"], c["ny"], c["nx"])
    W = torch.empty((5,) + n, dtype=torch.float64, device="cuda")
    if c["flow"] == "turbulence":
        # random solenoidal velocity with spectrum k^4 exp(-2 (k/4)^2), u_rms = 1; rho = T = 1
        k = torch.meshgrid(*[wave_numbers(m) for m in n], indexing="ij")[::-1]
        k2 = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
        amp = torch.sqrt(k2 * torch.exp(-k2 / 8.0))
        hat = [torch.fft.fftn(torch.randn(n, dtype=torch.float64, device="cuda", generator=g)) * amp for _ in range(3)]
        along = sum(a * b for a, b in zip(k, hat)) / k2.clamp(min=1.0)
        for q in range(3):
            W[1 + q] = torch.fft.ifftn(hat[q] - k[q] * along).real
        W[1:4] /= torch.sqrt((W[1:4] ** 2).sum(0).mean() / 3.0)
        W[0] = 1.0
        W[4] = 1.0 / (GAMMA * mach(c) ** 2)
        return W
    r = lambda *s: torch.rand(*s, dtype=torch.float64, device="cuda", generator=g)
    x = [(torch.arange(m, dtype=torch.float64, device="cuda") + 0.5) / m for m in n]
    z, y, x = torch.meshgrid(*x, indexing="ij")
    if c["flow"] == "pulse":
        # a smooth stream with a pressure pulse and a few random modes
        p0 = 1.0 / (GAMMA * mach(c) ** 2)
        a, ph, cx = r(5, 3), r(5, 3) * 2 * math.pi, 0.3 + 0.4 * r(3)
        for q in range(5):
            W[q] = sum(a[q, m] * torch.sin(2 * math.pi * (m + 1) * s + ph[q, m]) for m, s in enumerate((x, y, z))) / 3.0
        bump = torch.exp(-60.0 * ((x - cx[0]) ** 2 + (y - cx[1]) ** 2 + (z - cx[2]) ** 2))
        W[0] = 1.0 + 0.1 * W[0] + 0.2 * bump
        W[1] += 0.5
        W[4] = p0 * (1.0 + 0.05 * W[4] + 0.3 * bump)
        return W
    # four constant states about (0.5, 0.5), each a few per cent off the solver's own
    f = 1.0 + 0.04 * (r(4, 2) - 0.5)
    hi_x, hi_y = x >= 0.5, y >= 0.5
    four = [(hi_x & hi_y, (1.1, 0.0, 0.0, 1.1)), (~hi_x & hi_y, (0.5065, 0.8939, 0.0, 0.35)),
            (~hi_x & ~hi_y, (1.1, 0.8939, 0.8939, 1.1)), (hi_x & ~hi_y, (0.5065, 0.0, 0.8939, 0.35))]
    W.zero_()
    for m, (where, (rho, u, v, p)) in enumerate(four):
        for q, s in ((0, rho * f[m, 0]), (1, u), (2, v), (4, p * f[m, 1])):
            W[q] = torch.where(where, s, W[q])
    return W


def tubes(c, seed):
    """(grids, left states, right states, end times); the grids are the case's, the rest comes from the seed."""
    n = c["tubes"]
    nx = np.random.default_rng(n).choice(TUBES, size=n)
    rng = np.random.default_rng(seed)
    side = lambda: np.stack([rng.uniform(0.1, 1.0, n), rng.uniform(-1, 1, n), rng.uniform(0.1, 3.5, n)], axis=1)
    left, right = side(), side()
    grids = [GridDesc(global_nx=int(m), global_ny=c["ny"], global_nz=c["nz"], Lx=1.0, Ly=1.0, Lz=1.0) for m in nx]
    return grids, left, right, rng.uniform(0.14, 0.2, n)


def tube_state(m, ny, nz, left, right):
    lo = (np.arange(m) / m < 0.5)[None, None, :]
    one = np.ones((nz, ny, m))
    rho, u, p = (np.where(lo, left[q], right[q]) * one for q in range(3))
    return rho, u, 0 * one, 0 * one, p


def prepare(c, seed):
    P, G = params(dict(c, nx=16, ny=4, nz=4) if c["kind"] == "batch" else c)
    if c["kind"] == "batch":
        grids, left, right, t_end = tubes(c, seed)
        b = Batch(P, grids, t_end)
        for i, g in enumerate(grids):
            b.set_interior_primitives(i, *tube_state(g.global_nx, c["ny"], c["nz"], left[i], right[i]))
        b.set_config(0, 256, 1)  # the schedule that the autotuner picks for such a batch
        return {"case": c, "batch": b}
    s = Solver(P, G)
    s.set_interior_primitives(*fields(c, seed).cpu().numpy())
    st = {"case": c, "solver": s}
    if c["kind"] == "vjp":
        st["ubar"] = np.random.default_rng(seed).standard_normal((5,) + s.shape)
    return st


# ------------------------------------------------------------------ the pass

def run(st):
    c = st["case"]
    if c["kind"] == "batch":
        b = st["batch"]
        b.run(c["steps"])
        W = [b.primitives(i) for i in range(len(b.grids))]
        return {"fields": list(np.concatenate([w.reshape(5, -1) for w in W], axis=1)),
                "interior": list(np.concatenate([w[:, 3:-3, 3:-3, 3:-3].reshape(5, -1) for w in W], axis=1))}
    s = st["solver"]
    if c["kind"] == "vjp":
        return {"ubar": list(s.vjp_rk3_step(c["dt"], st["ubar"]))}
    if c["kind"] == "adjoint":
        J, grad, _ = s.adjoint_kinetic_energy(c["steps"], c["dt"], c["every"])
        return {"J": J, "grad": list(grad)}
    out = {}
    if c["kind"] == "step":
        if c["monitor"]:
            s.compute_rhs()
            out["rhs"] = [v[3:-3, 3:-3, 3:-3].clone() for v in s.device_view(RHS)]
        for _ in range(c["steps"]):
            out["dt"] = s.compute_timestep()
            s.rk3_step(out["dt"])
    elif c["kind"] == "fixed":
        s.rk3_steps(c["steps"], c["dt"])
    else:
        out["time"], _ = s.time_advance(1e9, c["steps"])
    if c["monitor"]:
        out["residuals"] = s.residuals()
        out["energy"] = s.total_energy()
        d = s.diagnostics()
        out["dissipation"], out["u_rms"] = d["dissipation"], d["u_rms"]
    out["fields"] = views(s, PRIMITIVE)  # every cell, ghosts among them
    out["interior"] = views(s, PRIMITIVE, interior=True)
    return out


def views(s, what, interior=False):
    """The resident arrays of a group, which keep their solver alive as long as they are used."""
    found = [v[3:-3, 3:-3, 3:-3] if interior else v for v in s.device_view(what)]
    for v in found:
        v.solver = s
    return found


# --------------------------------------------------------------------- work

def work(c):
    """One pass: each state array read once and written once; the operations of its formulas."""
    if c["kind"] == "batch":
        cells = c["tubes"] * (sum(TUBES) / len(TUBES)) * c["ny"] * c["nz"]
    else:
        cells = c["nx"] * c["ny"] * c["nz"]
    word = 4 if c["mixed"] else 8
    side = {WENO5: 52, LINEAR: 11, HYBRID: 21}[c["interp"]] + (50 if c["char"] else 0)
    rhs = 3 * (10 * side + {ROE: 150, HLLC: 110, HLL: 90, RUSANOV: 80}[c["riemann"]] + 45 + 15)
    if math.isfinite(c["re"]):
        rhs += 12 * 11 + 70 + 3 * 4 * 12
    step = 3 * (rhs + 5 * 5 + 25)
    if c["kind"] == "vjp":
        return {"bytes": cells * 5 * 8 * 3, "flops": cells * 3 * step}  # stage states, then the reverse of each
    if c["kind"] == "adjoint":
        last = c["steps"] - c["every"] * ((c["steps"] - 1) // c["every"])
        return {"bytes": cells * 8 * 8, "flops": cells * step * (3 * c["steps"] + (c["steps"] - last))}
    return {"bytes": cells * 10 * word, "flops": cells * (step * c["steps"] + (rhs if c["kind"] == "step" and c["monitor"] else 0))}


# -------------------------------------- the same in 64 bits, in plain torch

def cut(a, d, lo, hi):
    """Points lo .. hi - 1 of axis d."""
    return a.narrow(d, lo, hi - lo)


def pad(W, d, lo, hi, ng=3):
    """W (..., 5, z, y, x) with ng ghost cells either side of axis d (negative); boundary types lo, hi."""
    n = W.shape[d]
    if lo == hi == PERIODIC:
        return torch.cat([cut(W, d, n - ng, n), W, cut(W, d, 0, ng)], d)
    sign = torch.ones(5, 1, 1, 1, dtype=W.dtype, device=W.device)
    sign[-d] = -1.0  # axis -1 (x): velocity 1; -2 (y): 2; -3 (z): 3
    first, last = cut(W, d, 0, 1), cut(W, d, n - 1, n)
    a = torch.cat([first] * ng, d) if lo == OUTFLOW else cut(W, d, 0, ng).flip(d) * sign
    b = torch.cat([last] * ng, d) if hi == OUTFLOW else cut(W, d, n - ng, n).flip(d) * sign
    return torch.cat([a, W, b], d)


def to_cons(W):
    r, u, v, w, p = W.unbind(-4)
    return torch.stack([r, r * u, r * v, r * w, p / (GAMMA - 1) + 0.5 * r * (u * u + v * v + w * w)], -4)


def to_prim(U):
    r = torch.where(U.select(-4, 0) <= 0, torch.full_like(U.select(-4, 0), 1e-12), U.select(-4, 0))
    u, v, w = (U.select(-4, q) / r for q in (1, 2, 3))
    return torch.stack([r, u, v, w, (GAMMA - 1) * (U.select(-4, 4) - 0.5 * r * (u * u + v * v + w * w))], -4)


def weno5(f0, f1, f2, f3, f4):
    b = [13 / 12 * (f0 - 2 * f1 + f2) ** 2 + 0.25 * (f0 - 4 * f1 + 3 * f2) ** 2,
         13 / 12 * (f1 - 2 * f2 + f3) ** 2 + 0.25 * (f1 - f3) ** 2,
         13 / 12 * (f2 - 2 * f3 + f4) ** 2 + 0.25 * (3 * f2 - 4 * f3 + f4) ** 2]
    a = [d / (1e-6 + x) ** 2 for d, x in zip((1 / 16, 5 / 8, 5 / 16), b)]
    p = (3 * f0 - 10 * f1 + 15 * f2) / 8, (-f1 + 6 * f2 + 3 * f3) / 8, (3 * f2 + 6 * f3 - f4) / 8
    return (a[0] * p[0] + a[1] * p[1] + a[2] * p[2]) / (a[0] + a[1] + a[2])


DISP, DISS = 0.0463783, 0.01


def linear6(f):
    c = ((3 * DISP + 3 * DISS) / 8, (-18 * DISP - 30 * DISS - 1) / 16, (12 * DISP + 60 * DISS + 9) / 16,
         (12 * DISP - 60 * DISS + 9) / 16, (-18 * DISP + 30 * DISS - 1) / 16, (3 * DISP - 3 * DISS) / 8)
    return sum(a * b for a, b in zip(c, f))


def mdcd_nonlinear(f):
    f0, f1, f2, f3, f4, f5 = f
    b0 = 13 / 12 * (f0 - 2 * f1 + f2) ** 2 + 0.25 * (f0 - 4 * f1 + 3 * f2) ** 2
    b1 = 13 / 12 * (f1 - 2 * f2 + f3) ** 2 + 0.25 * (f1 - f3) ** 2
    b2 = 13 / 12 * (f2 - 2 * f3 + f4) ** 2 + 0.25 * (3 * f2 - 4 * f3 + f4) ** 2
    b3 = (271799 * f0 * f0 + f0 * (-2380800 * f1 + 4086352 * f2 - 3462252 * f3 + 1458762 * f4 - 245620 * f5)
          + f1 * (5653317 * f1 - 20427884 * f2 + 17905032 * f3 - 7727988 * f4 + 1325006 * f5)
          + f2 * (19510972 * f2 - 35817664 * f3 + 15929912 * f4 - 2792660 * f5)
          + f3 * (17195652 * f3 - 15880404 * f4 + 2863984 * f5) + f4 * (3824847 * f4 - 1429976 * f5)
          + 139633 * f5 * f5) / 120960
    tau = (b3 - (b0 + 4 * b1 + b2) / 6).abs()
    d = (1.5 * (DISP + DISS), 0.5 - 1.5 * (DISP - 3 * DISS), 0.5 - 1.5 * (DISP + 3 * DISS), 1.5 * (DISP - DISS))
    a = [w * (20 + tau / (x + 1e-40)) ** 2 for w, x in zip(d, (b0, b1, b2, b3))]
    q = (3 * f0 - 10 * f1 + 15 * f2, -f1 + 6 * f2 + 3 * f3, 3 * f2 + 6 * f3 - f4, 15 * f3 - 10 * f4 + 3 * f5)
    return sum(x * y for x, y in zip(a, q)) / (8 * (a[0] + a[1] + a[2] + a[3]))


def smooth_at(fm2, fm1, f0, fp1, fp2):
    eps = 0.9 * 0.4 / (1 - 0.9 * 0.4) * 1e-4
    a = (f0 - fm1).abs() + (f0 - 2 * fm1 + fm2).abs()
    b = (f0 - fp1).abs() + (f0 - 2 * fp1 + fp2).abs()
    return (2 * a * b + eps) / (a * a + b * b + eps) > 0.4


def interpolate(f, kind):
    """Left-biased midpoint value from the six points of a face's stencil."""
    if kind == WENO5:
        return weno5(*f[:5])
    if kind == LINEAR:
        return linear6(f)
    return torch.where(smooth_at(*f[:5]) & smooth_at(*f[1:]), linear6(f), mdcd_nonlinear(f))


def eigen(W, d):
    """Left and right eigenvectors (lists of rows) of the flux Jacobian along velocity d of primitives W (list)."""
    r, u, v, w, p = W
    nx, ny, nz = (1.0 if d == m else 0.0 for m in (1, 2, 3))
    g1 = GAMMA - 1
    q2 = u * u + v * v + w * w
    c = torch.sqrt(GAMMA * p / r)
    V, phi = nx * u + ny * v + nz * w, 0.5 * g1 * q2
    s2 = math.sqrt(2.0)
    a2, a3, a4, a5, a6, ic2 = 1 / (s2 * r * c), r / (s2 * c), (phi + c * c) / g1, 1 - phi / (c * c), phi / g1, 1 / (c * c)
    L = [[a2 * (phi + c * V), -a2 * (g1 * u + nx * c), -a2 * (g1 * v + ny * c), -a2 * (g1 * w + nz * c), g1 * a2],
         [nx * a5 - (nz * v - ny * w) / r, nx * g1 * u * ic2, nx * g1 * v * ic2 + nz / r, nx * g1 * w * ic2 - ny / r, -nx * g1 * ic2],
         [nz * a5 - (ny * u - nx * v) / r, nz * g1 * u * ic2 + ny / r, nz * g1 * v * ic2 - nx / r, nz * g1 * w * ic2, -nz * g1 * ic2],
         [ny * a5 - (nx * w - nz * u) / r, ny * g1 * u * ic2 - nz / r, ny * g1 * v * ic2, ny * g1 * w * ic2 + nx / r, -ny * g1 * ic2],
         [a2 * (phi - c * V), -a2 * (g1 * u - nx * c), -a2 * (g1 * v - ny * c), -a2 * (g1 * w - nz * c), g1 * a2]]
    R = [[a3, nx, nz, ny, a3],
         [a3 * (u - nx * c), nx * u, nz * u + ny * r, ny * u - nz * r, a3 * (u + nx * c)],
         [a3 * (v - ny * c), nx * v + nz * r, nz * v - nx * r, ny * v, a3 * (v + ny * c)],
         [a3 * (w - nz * c), nx * w - ny * r, nz * w, ny * w + nx * r, a3 * (w + nz * c)],
         [a3 * (a4 - c * V), nx * a6 + r * (nz * v - ny * w), nz * a6 + r * (ny * u - nx * v), ny * a6 + r * (nx * w - nz * u),
          a3 * (a4 + c * V)]]
    return L, R


def flux_of(U, d):
    r = U[0]
    u = [U[m] / r for m in (1, 2, 3)]
    p = (GAMMA - 1) * (U[4] - 0.5 * r * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2))
    un = u[d - 1]
    F = [r * un, U[1] * un, U[2] * un, U[3] * un, (U[4] + p) * un]
    F[d] = F[d] + p
    return F, u, p, un, torch.sqrt(GAMMA * p / r)


def riemann(UL, UR, d, kind):
    FL, uL, pL, nL, aL = flux_of(UL, d)
    FR, uR, pR, nR, aR = flux_of(UR, d)
    if kind == ROE:
        sL, sR = torch.sqrt(UL[0]), torch.sqrt(UR[0])
        mean = lambda x, y: (sL * x + sR * y) / (sL + sR)
        u = [mean(x, y) for x, y in zip(uL, uR)]
        H = mean((UL[4] + pL) / UL[0], (UR[4] + pR) / UR[0])
        q2 = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
        c2 = (GAMMA - 1) * (H - 0.5 * q2)
        c, V = torch.sqrt(c2), u[d - 1]
        dU = [y - x for x, y in zip(UL, UR)]
        t = 0.5 * (GAMMA - 1) * q2 * dU[0] + (GAMMA - 1) * (dU[4] - u[0] * dU[1] - u[1] * dU[2] - u[2] * dU[3])
        s = c * (V * dU[0] - dU[d])
        lam = [(V - c).abs(), V.abs(), (V + c).abs()]
        delta = 0.1 * (lam[1] + c)
        lam = [torch.where(x < delta, (x * x + delta * delta) / (2 * delta), x) for x in lam]
        k0, k4 = (lam[0] - lam[1]) * (t + s) / (2 * c2), (lam[2] - lam[1]) * (t - s) / (2 * c2)
        D = [lam[1] * dU[0] + k0 + k4] + [lam[1] * dU[m] + (k0 + k4) * u[m - 1] for m in (1, 2, 3)]
        D[d] = D[d] + c * (k4 - k0)
        D.append(lam[1] * dU[4] + k0 * (H - c * V) + k4 * (H + c * V))
        return [0.5 * (x + y - z) for x, y, z in zip(FL, FR, D)]
    SL, SR = torch.minimum(nL - aL, nR - aR), torch.maximum(nL + aL, nR + aR)
    if kind == HLL:
        mid = [(SR * f - SL * g + SL * SR * (y - x)) / (SR - SL) for f, g, x, y in zip(FL, FR, UL, UR)]
    else:
        dL, dR = UL[0] * (SL - nL), UR[0] * (SR - nR)
        SM = (dR * nR - dL * nL + pL - pR) / (dR - dL)

        def star(U, F, u, p, n, S):
            rs = U[0] * (S - n) / (S - SM)
            v = [SM if m == d - 1 else u[m] for m in range(3)]
            e = U[4] / U[0] + (SM - n) * (SM + p / (U[0] * (S - n)))
            return [f + S * (rs * x - y) for f, x, y in zip(F, [1.0] + v + [e], U)]
        mid = [torch.where(SM >= 0, x, y) for x, y in zip(star(UL, FL, uL, pL, nL, SL), star(UR, FR, uR, pR, nR, SR))]
    return [torch.where(SL >= 0, f, torch.where(SR <= 0, g, m)) for f, g, m in zip(FL, FR, mid)]


def derivative(f, d, h, per):
    """First derivative along axis d: 6th order, with the solver's one-sided and reduced orders at a boundary
    (its right-hand one-sided form is -df/dx)."""
    n = f.shape[d]
    g = torch.cat([cut(f, d, n - 3, n), f, cut(f, d, 0, 3)], d)
    at = lambda o: g.narrow(d, 3 + o, n)
    out = (at(3) - 9 * at(2) + 45 * at(1) - 45 * at(-1) + 9 * at(-2) - at(-3)) / (60 * h)
    if per:
        return out
    col = [f.select(d, m) for m in range(5)] + [f.select(d, n - 1 - m) for m in range(5)]
    two = lambda a: (-3 * a[0] + 4 * a[1] - a[2]) / (2 * h)
    lo = [two(col[:3]), (col[2] - col[0]) / (2 * h), (-col[4] + 8 * col[3] - 8 * col[1] + col[0]) / (12 * h)]
    e = col[5:]
    hi = [(-e[0] + 8 * e[1] - 8 * e[3] + e[4]) / (12 * h), (e[0] - e[2]) / (2 * h), two(e[:3])]
    return torch.cat([torch.stack(lo, d), cut(out, d, 3, n - 3), torch.stack(hi, d)], d)


def rhs_of(W, c, h):
    """-div F + viscous terms of primitives W (..., 5, z, y, x)."""
    bc = [int(x) for x in c["bc"]]
    R = 0.0
    for d, axis in ((1, -1), (2, -2), (3, -3)):
        lo, hi = bc[2 * d - 2], bc[2 * d - 1]
        per = lo == hi == PERIODIC
        n = W.shape[axis]
        Wp = pad(W, axis, lo, hi)
        Up = to_cons(Wp)
        cells = lambda A, m: [x.narrow(axis, m, n + 1) for x in A.unbind(-4)]  # of the face's stencil, point m
        st = [cells(Up, m) for m in range(6)]
        if c["char"]:
            sides = []
            for base, order in ((2, range(6)), (3, range(5, -1, -1))):
                L, Rm = eigen(cells(Wp, base), d)
                q = [interpolate([sum(L[r][s] * st[m][s] for s in range(5)) for m in order], c["interp"]) for r in range(5)]
                sides.append([sum(Rm[r][s] * q[s] for s in range(5)) for r in range(5)])
            UL, UR = sides
        else:
            UL = [interpolate([st[m][q] for m in range(6)], c["interp"]) for q in range(5)]
            UR = [interpolate([st[5 - m][q] for m in range(6)], c["interp"]) for q in range(5)]
        del st
        F = torch.stack(riemann(UL, UR, d, c["riemann"]), -4)  # faces -1/2 .. n - 1/2
        if per:
            F = torch.cat([cut(F, axis, n - 2, n), F, cut(F, axis, 1, 3)], axis)
        else:
            ends = [torch.cat([e if t == OUTFLOW else torch.zeros_like(e)] * 2, axis)
                    for e, t in ((cut(F, axis, 0, 1), lo), (cut(F, axis, n, n + 1), hi))]
            F = torch.cat([ends[0], F, ends[1]], axis)
        f = [F.narrow(axis, m, n) for m in range(6)]
        R = R - ((f[3] - f[2]) * (75 / 64) - (f[4] - f[1]) * (25 / 384) + (f[5] - f[0]) * (3 / 640)) / h[d - 1]
    if math.isfinite(c["re"]):
        R = R + viscous(W, c, h, bc)
    return R


def viscous(W, c, h, bc):
    Ma, S = mach(c), 110.4 / 273.15
    Rgas = 1 / (GAMMA * Ma * Ma)
    r, u, v, w, p = W.unbind(-4)
    T = p / (r * Rgas)
    per = [bc[2 * m] == bc[2 * m + 1] == PERIODIC for m in range(3)]
    D = lambda f, m: derivative(f, -1 - m, h[m], per[m])
    G = [[D(f, m) for m in range(3)] for f in (u, v, w, T)]
    mu = T ** 1.5 * (1 + S) / (T + S) / c["re"]
    kappa = mu * GAMMA * Rgas / (GAMMA - 1) / 0.72
    div = G[0][0] + G[1][1] + G[2][2]
    tau = [[mu * (G[a][b] + G[b][a]) - (2 / 3 * mu * div if a == b else 0.0) for b in range(3)] for a in range(3)]
    out = [torch.zeros_like(r)]
    for a in range(3):
        out.append(D(tau[a][0], 0) + D(tau[a][1], 1) + D(tau[a][2], 2))
    e = [u * tau[0][m] + v * tau[1][m] + w * tau[2][m] + kappa * G[3][m] for m in range(3)]
    out.append(D(e[0], 0) + D(e[1], 1) + D(e[2], 2))
    return torch.stack(out, -4)


def rk3(U, dt, c, h):
    L = lambda V: rhs_of(to_prim(V), c, h)
    U1 = U + dt * L(U)
    U2 = 0.75 * U + 0.25 * (U1 + dt * L(U1))
    return U / 3 + 2 / 3 * (U2 + dt * L(U2))


def speed_limit(U, dx):
    """dx / max(|u| + a) of each problem, the pressure from the x momentum alone as the solver has it."""
    r, u = U.select(-4, 0), U.select(-4, 1) / U.select(-4, 0)
    a = torch.sqrt(GAMMA * (GAMMA - 1) * (U.select(-4, 4) - 0.5 * r * u * u) / r)
    return dx / (u.abs() + a).amax(dim=(-3, -2, -1))


def energy_of(U, vol):
    return 0.5 * ((U[1:4] ** 2).sum(0) / U[0]).sum() * vol


def exact(c, seed):
    with torch.no_grad():
        if c["kind"] == "batch":
            return exact_tubes(c, seed)
        h = [l / n for l, n in zip(lengths(c), (c["nx"], c["ny"], c["nz"]))]
        W = fields(c, seed)
        if c["kind"] in ("vjp", "adjoint"):
            return exact_reverse(c, W, h, seed)
        U, out, t, before = to_cons(W), {}, 0.0, None
        if c["kind"] == "step" and c["monitor"]:
            out["rhs"] = list(rhs_of(W, c, h))
        for _ in range(c["steps"]):
            dt = c["dt"] if c["kind"] == "fixed" else float(0.4 * speed_limit(U, h[0]))
            t += dt
            before = U
            U = rk3(U, dt, c, h)
        if c["kind"] == "step":
            out["dt"] = dt
        elif c["kind"] == "advance":
            out["time"] = t
        W = to_prim(U)
        if c["monitor"]:
            vol = h[0] * h[1] * h[2]
            out["residuals"] = torch.stack([torch.sqrt(((a - b) ** 2).sum() * h[0] ** 3) / a.abs().max()
                                            for a, b in zip(U, before)]).cpu().numpy()
            out["energy"] = float(energy_of(U, vol))
            out["dissipation"], out["u_rms"] = dissipation(W, c, h)
        out["fields"] = None
        out["interior"] = list(W)
        return out


def dissipation(W, c, h):
    bc = [int(x) for x in c["bc"]]
    S, Rgas = 110.4 / 273.15, 1 / (GAMMA * mach(c) ** 2)
    T = W[4] / (W[0] * Rgas)
    mu = (T ** 1.5 * (1 + S) / (T + S)).mean() / c["re"] if math.isfinite(c["re"]) else torch.zeros(())
    g2 = sum((derivative(W[1 + a], -1 - m, h[m], bc[2 * m] == bc[2 * m + 1] == PERIODIC) ** 2).mean()
             for a in range(3) for m in range(3))
    return float(mu / W[0].mean() * g2), float(torch.sqrt((W[1:4] ** 2).sum(0).mean() / 3))


def exact_reverse(c, W, h, seed):
    def back(U, ubar):
        with torch.enable_grad():
            V = U.detach().requires_grad_()
            (g,) = torch.autograd.grad(rk3(V, c["dt"], c, h), V, ubar)
        return g
    U = [to_cons(W)]
    if c["kind"] == "vjp":
        ubar = torch.from_numpy(np.random.default_rng(seed).standard_normal((5, c["nz"] + 6, c["ny"] + 6, c["nx"] + 6)))
        out = torch.zeros_like(ubar)
        out[:, 3:-3, 3:-3, 3:-3] = back(U[0], ubar[:, 3:-3, 3:-3, 3:-3].cuda()).cpu()
        return {"ubar": list(out.numpy())}
    for _ in range(c["steps"]):
        U.append(rk3(U[-1], c["dt"], c, h))
    vol = h[0] * h[1] * h[2]
    end = U.pop()
    J = float(energy_of(end, vol))
    u = end[1:4] / end[0]
    ubar = vol * torch.cat([-0.5 * (u * u).sum(0, keepdim=True), u, torch.zeros_like(end[4:])])
    for V in reversed(U):
        ubar = back(V, ubar)
    # U = (rho, rho u, ..., p/(g-1) + rho |u|^2 / 2) at fixed rho and p
    return {"J": J, "grad": list((W[0] * (ubar[1:4] + ubar[4] * W[1:4])).cpu().numpy())}


def exact_tubes(c, seed):
    grids, left, right, t_end = tubes(c, seed)
    found = [None] * len(grids)
    for m in sorted({g.global_nx for g in grids}):
        which = [i for i, g in enumerate(grids) if g.global_nx == m]
        W = torch.from_numpy(np.stack([np.stack(tube_state(m, c["ny"], c["nz"], left[i], right[i])) for i in which])).cuda()
        h = (1.0 / m, 1.0 / c["ny"], 1.0 / c["nz"])
        U, t = to_cons(W), torch.zeros(len(which), dtype=torch.float64, device="cuda")
        end = torch.from_numpy(t_end[which]).cuda()
        for _ in range(c["steps"]):
            dt = torch.minimum(0.4 * speed_limit(U, h[0]), end - t)
            t = t + dt
            U = rk3(U, dt[:, None, None, None, None], c, h)
        for k, i in enumerate(which):
            found[i] = to_prim(U[k]).cpu().numpy()
    return {"fields": None, "interior": [np.concatenate([w[q].reshape(-1) for w in found]) for q in range(5)]}
