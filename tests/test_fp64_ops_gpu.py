"""The branch-free FP64 quotients of the state conversions against IEEE
arithmetic, bit for bit: the conserved state of an uploaded field and the
state after an RK3 step of size zero (conversions to and fro in every stage)
equal numpy's unfused double arithmetic, over twelve decades of density and
pressure."""
import numpy as np
import pytest

from ns3d_wcns_b200.config import make_params

pytestmark = pytest.mark.gpu

N = (37, 22, 19)


def wide_state(shape, seed):
    rng = np.random.default_rng(seed)
    rho = 10.0 ** rng.uniform(-6, 6, shape)
    u, v, w = (rng.uniform(-3, 3, shape) for _ in range(3))
    p = 10.0 ** rng.uniform(-6, 6, shape)
    return [rho, u, v, w, p]


def to_cons(W, g):
    r, u, v, w, p = W
    kin = 0.5 * ((u * u + v * v) + w * w)
    return [r, r * u, r * v, r * w, r * (p / ((g - 1.0) * r) + kin)]


def to_prim(U, g):
    r = U[0]
    u, v, w = U[1] / r, U[2] / r, U[3] / r
    e = U[4] / r - 0.5 * ((u * u + v * v) + w * w)
    return [r, u, v, w, ((g - 1.0) * r) * e]


def test_conserved_bits(gpu_lib):
    from ns3d_wcns_b200.solver import Solver
    P, G = make_params(n=N, interpolation=0, riemann=0)
    with Solver(P, G) as s:
        W = wide_state(s.shape, 1)
        s.upload_primitives(W)
        for a, b in zip(s.conserved(), to_cons(W, P.gamma)):
            assert np.array_equal(a, b)


def test_stage_round_trip_bits(gpu_lib):
    from ns3d_wcns_b200 import _lib
    from ns3d_wcns_b200.slab import device_planes
    from ns3d_wcns_b200.solver import Solver
    P, G = make_params(n=N, Re=400.0, interpolation=2, riemann=2)
    with Solver(P, G) as s:
        rng = np.random.default_rng(2)
        n = tuple(reversed(N))
        W0 = [1.0 + 0.3 * rng.uniform(-1, 1, n), *(rng.uniform(-1, 1, n) for _ in range(3)), 8.0 + rng.uniform(-1, 1, n)]
        s.set_interior_primitives(*W0)
        s.rk3_step(0.0)
        inner = (slice(3, -3),) * 3
        U0 = to_cons(W0, P.gamma)
        W1 = to_prim(U0, P.gamma)                                           # U1 = U0 + 0
        W2 = to_prim([0.75 * a + 0.25 * b for a, b in zip(U0, to_cons(W1, P.gamma))], P.gamma)
        W3 = to_prim([(1.0 / 3.0) * a + (2.0 / 3.0) * b for a, b in zip(U0, to_cons(W2, P.gamma))], P.gamma)
        Rgas = 1.0 / (P.Ma * P.Ma * P.gamma)
        lay = s.device_fields(_lib.NS3D_TEMPERATURE)[1]
        T = device_planes(s, 0, N[2])[5].cpu().numpy().reshape(N[2], lay[1], lay[3])[:, 3:-3, 3:3 + N[0]]
        for a, b in zip(s.primitives(), W3):
            assert np.array_equal(a[inner], b)
        assert np.array_equal(T, W3[4] / (W3[0] * Rgas))
