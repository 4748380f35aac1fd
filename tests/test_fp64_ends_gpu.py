"""The FP64 conversions at the ends of the range against IEEE arithmetic, bit
for bit and with the sign of zero: conserved states of uploaded primitives
(both paths), and the mixed path's primitives recovered from them."""
import numpy as np
import pytest

from ns3d_wcns_b200.config import make_params
from test_fp64_ops_gpu import N, to_cons, to_prim, wide_state

pytestmark = pytest.mark.gpu

RHO = [np.inf, 4e307, 1e300, 1.0, 1e-5, 1e-300, 1e-310]
VEL = [0.0, -0.0, 0.5, -3.0, np.inf]
P_ = [np.inf, 1.5e308, 1e300, 2.0, 0.0, -0.0, 1e-280]


def ends(shape):
    """Every density with every pressure and velocity, and wide_state beyond them."""
    W = [a.reshape(-1).copy() for a in wide_state(shape, 6)]
    k = 0
    for r in RHO:
        for p in P_:
            for v in VEL:
                for q, x in enumerate((r, 0.25, v, -0.0, p)):
                    W[q][k] = x
                k += 1
    return [a.reshape(shape) for a in W]


def same(a, b):
    nan = np.isnan(a) & np.isnan(b)
    return np.array_equal(np.where(nan, 0, a).view(np.uint64), np.where(nan, 0, b).view(np.uint64))


@pytest.mark.parametrize("precision", [0, 1])
def test_conversion_ends(gpu_lib, precision):
    from ns3d_wcns_b200.solver import Solver
    P, G = make_params(n=N, interpolation=0, riemann=0, precision=precision)
    with Solver(P, G) as s, np.errstate(all="ignore"):
        W = ends(s.shape)
        U = to_cons(W, P.gamma)
        s.upload_primitives(W)
        for a, b in zip(s.conserved(), U):
            assert same(a, b)
        if precision:
            for a, b in zip(s.primitives(), to_prim(U, P.gamma)):
                assert same(a, b)
