"""The mixed path's FP32 rounding, which MDCD_HYBRID's detector turns into one
trajectory or another.

test_mixed_bits: the right-hand side and the primitives after two steps, bit
for bit against digests of the kernels that carried a face per thread through
shared memory (golden/mixed_bits.json), through the line kernel (small grids)
and the marching kernel, with two lines in a float2 (even line counts) and
with one.  MDCD_LINEAR, which has no detector, with HLLC on pairs, the form
both have; on single lines its HLLC has less error now.

test_hybrid_against_oracle: the right-hand side against the FP64 oracle on
under-resolved states whose warps have few and many faces in doubt.  Where no
detector flips, it is off by FP32 rounding: the states and the flux pass some
forty roundings on the way to a face, so 40 * 2^-24 of the largest flux, taken
through the difference's coefficients over h.  A flip moves its cells by more;
as many cells may be beyond the bound as four times those that the oracle
itself moves when its inputs are off by one FP32 unit, and twenty."""
import hashlib
import json
import os

import numpy as np
import pytest

from helpers import interior
from ns3d_wcns_b200.config import make_params
from ns3d_wcns_b200.initial import random_state

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "mixed_bits.json")
SIZES = [(24, 20, 38), (23, 21, 38), (61, 33, 64), (96, 40, 80), (65, 40, 64)]
SCHEMES = [(2, 2, 0), (3, 2, 0), (3, 0, 0), (3, 3, 0), (3, 2, 1), (2, 4, 1)]  # interpolation, riemann, characteristic
BCS = {"periodic": (0,) * 6, "bounded": (1, 1, 2, 2, 3, 3)}


def state(n, smooth):
    """random_state, averaged `smooth` times over the neighbours (additions and products only: the same on every machine)."""
    f = [np.asarray(a) for a in random_state(n, seed=5, amp=0.2)]
    for _ in range(smooth):
        for d in range(3):
            f = [0.25 * (np.roll(a, 1, d) + np.roll(a, -1, d)) + 0.5 * a for a in f]
    return f


def mixed_params(n, scheme, bcs):
    return make_params(n=n, L=tuple(0.1 * m for m in n), interpolation=scheme[0], riemann=scheme[1], char_recon=scheme[2],
                       bcs=bcs, Re=300.0, precision=1)


def cases():
    for i, n in enumerate(SIZES):
        for j, sc in enumerate(SCHEMES):
            if sc == (2, 2, 0) and (n[0] | n[1]) & 1:
                continue
            b = ("periodic", "bounded")[(i + j) % 2]
            yield n, sc, b, (i + j) % 3


def key(n, sc, b, smooth):
    return "%dx%dx%d %d%d%d %s %d" % (*n, *sc, b, smooth)


def digests(n, sc, b, smooth):
    from ns3d_wcns_b200.solver import Solver
    P, G = mixed_params(n, sc, BCS[b])
    with Solver(P, G) as s:
        s.set_interior_primitives(*state(n, smooth))
        s.compute_rhs()
        out = [interior(s.rhs()).astype(np.float32)]
        for _ in range(2):
            s.rk3_step(2e-3)
        out.append(interior(s.primitives()).astype(np.float32))
    return [hashlib.sha256(np.ascontiguousarray(a).tobytes()).hexdigest() for a in out]


@pytest.mark.gpu
@pytest.mark.parametrize("case", list(cases()), ids=lambda c: key(*c).replace(" ", "-"))
def test_mixed_bits(gpu_lib, case):
    with open(GOLDEN) as f:
        want = json.load(f)[key(*case)]
    assert digests(*case) == want


def flux_scale(W, g, G):
    """Per variable: the largest flux, through the half-node difference of every direction."""
    rho, u, v, w, p = W
    e = p / (g - 1) + 0.5 * rho * (u * u + v * v + w * w)
    speed = np.sqrt(u * u + v * v + w * w) + np.sqrt(g * p / rho)
    top = [rho * speed, *(abs(rho * m) * speed + p for m in (u, v, w)), (e + p) * speed]
    h = sum(1.0 / d for d in (G.dx, G.dy, G.dz))
    return np.array([t.max() for t in top]) * 2 * (75 / 64 + 25 / 384 + 3 / 640) * h


def oracle_rhs(P, G, W):
    from oracle import oracle
    o = oracle.PortSolver(P, G)
    o.set_interior_prims(*W)
    o.compute_rhs()
    return interior(o.rhs())


@pytest.mark.gpu
@pytest.mark.parametrize("n", [(24, 20, 38), (23, 21, 38), (96, 40, 80), (65, 40, 64)], ids=str)
@pytest.mark.parametrize("smooth", [0, 1, 4])
def test_hybrid_against_oracle(gpu_lib, n, smooth):
    from ns3d_wcns_b200.solver import Solver
    P, G = mixed_params(n, (3, 2, 0), BCS["periodic"])
    W = [a.astype(np.float32).astype(np.float64) for a in state(n, smooth)]
    ref = oracle_rhs(P, G, W)
    bound = (40 * 2.0 ** -24 * flux_scale(W, P.gamma, G))[:, None, None, None]
    rng = np.random.default_rng(1)
    near = oracle_rhs(P, G, [a * (1 + 2.0 ** -23 * rng.integers(-1, 2, a.shape)) for a in W])
    flips = int((abs(near - ref) > bound).any(0).sum())
    with Solver(P, G) as s:
        s.set_interior_primitives(*W)
        s.compute_rhs()
        got = interior(s.rhs())
    assert int((abs(got - ref) > bound).any(0).sum()) <= 4 * flips + 20
