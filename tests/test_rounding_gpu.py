"""The rounding of the FP64 arithmetic against wider precision.

test_rhs_rounding: the right-hand side's error (2-norm) against the oracle in
80-bit arithmetic is no larger than that of the kernels with IEEE reciprocals,
quotients and square roots and the eigenvector matrices, measured once on the
same states; one per cent is left for the compiler's placement of fused
operations.  test_mixed_rounding: the mixed path's with the component-wise
schemes without a detector, no larger than of any kernels before."""
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


def rhs_error(n, scheme, precision):
    from ns3d_wcns_b200.solver import Solver
    from oracle import oracle
    P, G = make_params(n=n, L=tuple(0.1 * m for m in n), interpolation=scheme[0], riemann=scheme[1],
                       char_recon=scheme[2], Re=300.0, precision=precision)
    W = random_state(n, seed=5, amp=0.2)
    o = oracle.ExtendedSolver(P, G)
    o.set_interior_prims(*W)
    o.compute_rhs()
    want = interior(o.rhs())
    with Solver(P, G) as s:
        s.set_interior_primitives(*W)
        s.compute_rhs()
        off = interior(s.rhs()).astype(np.longdouble) - want
    return float(np.sqrt((off ** 2).sum() / (want ** 2).sum()))


@pytest.mark.parametrize("scheme", list(FORMER), ids=str)
def test_rhs_rounding(gpu_lib, scheme):
    assert rhs_error(N, scheme, 0) <= 1.01 * FORMER[scheme]


MIXED = {((24, 20, 38), (0, 0, 0)): 4.391e-7, ((24, 20, 38), (0, 2, 0)): 4.896e-7, ((24, 20, 38), (0, 3, 0)): 4.464e-7,
         ((24, 20, 38), (0, 1, 0)): 4.495e-7, ((23, 21, 38), (2, 2, 0)): 5.000e-7, ((24, 20, 38), (2, 2, 0)): 8.688e-7,
         ((24, 20, 38), (2, 3, 0)): 4.315e-7}


@pytest.mark.parametrize("case", list(MIXED), ids=str)
def test_mixed_rounding(gpu_lib, case):
    assert rhs_error(*case, 1) <= 1.01 * MIXED[case]


def line_rhs(U, g, h):
    """Inviscid WENO5 + Rusanov right-hand side of periodic lines U (..., 5, n) along x, in U's precision."""
    at = lambda k: np.roll(U, -k, -1)  # cell i + k

    def weno5(f):
        f0, f1, f2, f3, f4 = f
        c = np.longdouble(13) / 12
        b = [c * (f0 - 2 * f1 + f2) ** 2 + (f0 - 4 * f1 + 3 * f2) ** 2 / 4, c * (f1 - 2 * f2 + f3) ** 2 + (f1 - f3) ** 2 / 4,
             c * (f2 - 2 * f3 + f4) ** 2 + (3 * f2 - 4 * f3 + f4) ** 2 / 4]
        a = [d / (np.longdouble(1e-6) + x) ** 2 for d, x in zip((1, 10, 5), b)]
        p = (3 * f0 - 10 * f1 + 15 * f2, -f1 + 6 * f2 + 3 * f3, 3 * f2 + 6 * f3 - f4)
        return sum(x * y for x, y in zip(a, p)) / (8 * sum(a))

    def side(V):
        r, u = V[..., 0, :], V[..., 1, :] / V[..., 0, :]
        p = (g - 1) * (V[..., 4, :] - (V[..., 1, :] ** 2 + V[..., 2, :] ** 2 + V[..., 3, :] ** 2) / (2 * r))
        F = V * u[..., None, :]
        F[..., 1, :] += p
        F[..., 4, :] += p * u
        return F, np.where(u.real < 0, -u, u) + np.sqrt(g * p / r)
    L, R = weno5([at(k) for k in (-2, -1, 0, 1, 2)]), weno5([at(k) for k in (3, 2, 1, 0, -1)])
    (FL, sL), (FR, sR) = side(L), side(R)
    s = np.where(sL.real < sR.real, sR, sL)[..., None, :]
    F = (FL + FR) / 2 - s * (R - L) / 2  # face i + 1/2
    f = lambda k: np.roll(F, -k, -1)
    return -(np.longdouble(75) / 64 * (f(0) - f(-1)) - np.longdouble(25) / 384 * (f(1) - f(-2))
             + np.longdouble(3) / 640 * (f(2) - f(-3))) / h


def test_vjp_rounding(gpu_lib):
    """The reverse mode of a nearly uniform line, where the weights' derivatives take differences of nearly equal
    candidates, against complex-step derivatives in 80-bit arithmetic.  Differences of 1e-2 of the values, formed from
    differences, leave some hundred units of 2^-53: 3e-14 (formed from the candidates themselves: 1.2e-13)."""
    from ns3d_wcns_b200.solver import Solver
    n = 48
    P, G = make_params(n=(n, 4, 4), L=(4.8, 0.4, 0.4), interpolation=0, riemann=1, Re=float("inf"))
    rng = np.random.default_rng(4)
    base = (1.05, 0.3, -0.2, 0.1, 8.5)
    W = [np.broadcast_to(b * (1 + 0.01 * rng.uniform(-0.5, 0.5, n)), (4, 4, n)) for b in base]
    rbar = rng.uniform(-0.5, 0.5, (5, n))
    with Solver(P, G) as s:
        s.set_interior_primitives(*W)
        U = interior(s.conserved())[:, 0, 0, :]
        full = np.zeros((5,) + s.shape)
        full[:, 3:-3, 3:-3, 3:-3] = rbar[:, None, None, :]
        got = interior(s.vjp_rhs(full))[:, 1, 2, :]
    step = np.longdouble(1e-60)
    V = np.broadcast_to(U.astype(np.clongdouble), (5 * n, 5, n)).copy()
    V.reshape(5 * n, 5 * n)[np.arange(5 * n), np.arange(5 * n)] += 1j * step
    R = line_rhs(V, np.longdouble(P.gamma), np.longdouble(G.dx))
    want = ((R.imag / step) * rbar.astype(np.longdouble)).sum(axis=(1, 2)).reshape(5, n)
    assert float(np.sqrt(((got - want) ** 2).sum() / (want ** 2).sum())) <= 3e-14
