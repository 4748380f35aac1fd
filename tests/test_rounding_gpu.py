"""The rounding of the FP64 arithmetic against wider precision.

test_rhs_rounding: the right-hand side's error (2-norm) against the oracle in
80-bit arithmetic is no larger than that of the kernels with IEEE reciprocals,
quotients and square roots and the eigenvector matrices, measured once on the
same states; one per cent is left for the compiler's placement of fused
operations."""
import numpy as np
import pytest

from helpers import interior
from ns3d_wcns_b200.config import make_params
from ns3d_wcns_b200.initial import random_state

pytestmark = pytest.mark.gpu

N = (40, 36, 32)
FORMER = {(0, 0, 0): 1.118e-15, (0, 2, 0): 1.487e-15, (0, 3, 0): 1.120e-15, (2, 2, 0): 1.342e-15, (3, 2, 0): 1.649e-15,
          (3, 0, 0): 1.249e-15, (0, 1, 0): 1.134e-15, (2, 4, 0): 1.324e-15, (2, 5, 0): 9.265e-16,
          (0, 0, 1): 2.069e-15, (3, 2, 1): 2.495e-15, (0, 3, 1): 2.018e-15}  # interpolation, riemann, characteristic


@pytest.mark.parametrize("scheme", list(FORMER), ids=str)
def test_rhs_rounding(gpu_lib, scheme):
    from ns3d_wcns_b200.solver import Solver
    from oracle import oracle
    P, G = make_params(n=N, L=tuple(0.1 * m for m in N), interpolation=scheme[0], riemann=scheme[1],
                       char_recon=scheme[2], Re=300.0)
    W = random_state(N, seed=5, amp=0.2)
    o = oracle.ExtendedSolver(P, G)
    o.set_interior_prims(*W)
    o.compute_rhs()
    want = interior(o.rhs())
    with Solver(P, G) as s:
        s.set_interior_primitives(*W)
        s.compute_rhs()
        off = interior(s.rhs()).astype(np.longdouble) - want
    assert float(np.sqrt((off ** 2).sum() / (want ** 2).sum())) <= 1.01 * FORMER[scheme]

