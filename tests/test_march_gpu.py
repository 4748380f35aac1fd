"""The line-marching sweeps (y and z, one line per thread) where they can go
wrong: the smallest lines, line counts that leave a block partly empty, lines
cut into segments, and every boundary type, against the CPU oracle.
Tolerance: the FP64 path's own bounds, 1e-12 of the largest right-hand side
and 1e-10 of the state after two steps."""
import numpy as np
import pytest

from helpers import interior, rel_linf
from ns3d_wcns_b200.config import make_params
from ns3d_wcns_b200.initial import random_state
from oracle import oracle

pytestmark = pytest.mark.gpu

SIZES = [(3, 3, 3), (5, 4, 7), (21, 3, 6), (33, 70, 5), (6, 9, 130)]
BCS = [(0,) * 6, (3, 3, 1, 2, 4, 4), (1, 2, 3, 3, 0, 0)]


@pytest.mark.parametrize("n", SIZES, ids=str)
@pytest.mark.parametrize("bcs", BCS, ids=["periodic", "mixed", "z-periodic"])
@pytest.mark.parametrize("interp,rs", [(0, 0), (3, 2), (2, 2), (0, 2), (3, 0)])
def test_march_against_oracle(gpu_lib, n, bcs, interp, rs):
    from ns3d_wcns_b200.solver import Solver
    P, G = make_params(n=n, L=(1.0, 0.8, 0.9), interpolation=interp, riemann=rs, bcs=bcs, Re=300.0, dt_fixed=1e-4)
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
            s.rk3_step(1e-4)
            o.rk3_step(1e-4)
        for a, b in zip(interior(s.conserved()), interior(o.conserved())):
            assert rel_linf(a, b) <= 1e-10
