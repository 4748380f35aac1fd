"""The marching kernel at its edges, on grids that do take it (line_takes in
sweep_line.cuh: more than 3552 chunks of lines along y, 1776 along z; for
pairs in FP32 3552 and 1184): lines of 3 to 7 cells, line counts that leave a
block partly empty, lines cut into segments, every boundary type.  FP64
against the oracle with the path's own bounds, 1e-12 of the largest right-hand
side and 1e-10 of the state after two steps; mixed with test_mixed_bits_gpu's
bound (40 roundings of the largest flux, and the cells that a unit of FP32
flips in the oracle)."""
import numpy as np
import pytest

from helpers import interior, rel_linf
from ns3d_wcns_b200.config import make_params
from ns3d_wcns_b200.initial import random_state
from oracle import oracle
from test_mixed_bits_gpu import flux_scale, oracle_rhs

pytestmark = pytest.mark.gpu

ALONG_Y = [(120, 3, 31), (119, 5, 32), (61, 130, 61)]
ALONG_Z = [(60, 30, 3), (61, 31, 5), (45, 40, 7), (60, 31, 130)]
BCS = {"periodic": (0,) * 6, "mixed": (3, 3, 1, 2, 2, 1), "outflow": (1, 2, 3, 3, 3, 3)}


@pytest.mark.parametrize("n", ALONG_Y + ALONG_Z, ids=str)
@pytest.mark.parametrize("bcs", list(BCS))
@pytest.mark.parametrize("scheme", [(0, 0), (3, 2), (2, 2), (0, 3)], ids=str)
def test_fp64(gpu_lib, n, bcs, scheme):
    from ns3d_wcns_b200.solver import Solver
    P, G = make_params(n=n, L=tuple(0.1 * m for m in n), interpolation=scheme[0], riemann=scheme[1], bcs=BCS[bcs], Re=300.0)
    st = random_state(n, seed=5, amp=0.2)
    o = oracle.PortSolver(P, G)
    o.set_interior_prims(*st)
    o.compute_rhs()
    with Solver(P, G) as s:
        s.set_interior_primitives(*st)
        s.compute_rhs()
        for a, b in zip(interior(s.rhs()), interior(o.rhs())):
            assert rel_linf(a, b) <= 1e-12
        for _ in range(2):
            s.rk3_step(1e-3)
            o.rk3_step(1e-3)
        for a, b in zip(interior(s.conserved()), interior(o.conserved())):
            assert rel_linf(a, b) <= 1e-10


@pytest.mark.parametrize("n", [(120, 4, 62), (119, 5, 31), (60, 41, 4), (62, 40, 5), (61, 31, 4), (61, 31, 130)], ids=str)
@pytest.mark.parametrize("bcs", list(BCS))
@pytest.mark.parametrize("scheme", [(3, 2), (2, 2), (3, 0)], ids=str)
def test_mixed(gpu_lib, n, bcs, scheme):
    from ns3d_wcns_b200.solver import Solver
    P, G = make_params(n=n, L=tuple(0.1 * m for m in n), interpolation=scheme[0], riemann=scheme[1], bcs=BCS[bcs], Re=300.0,
                       precision=1)
    W = [a.astype(np.float32).astype(np.float64) for a in random_state(n, seed=5, amp=0.2)]
    ref = oracle_rhs(P, G, W)
    bound = (40 * 2.0 ** -24 * flux_scale(W, P.gamma, G))[:, None, None, None]
    rng = np.random.default_rng(1)
    near = oracle_rhs(P, G, [a * (1 + 2.0 ** -23 * rng.integers(-1, 2, a.shape)) for a in W])
    flips = int((abs(near - ref) > bound).any(0).sum())
    with Solver(P, G) as s:
        s.set_interior_primitives(*W)
        s.compute_rhs()
        got = interior(s.rhs())
    assert int((abs(got - ref) > bound).any(0).sum()) <= 4 * flips + (20 if scheme[0] == 3 else 0)
