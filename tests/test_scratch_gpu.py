"""What adjoint calls and batch downloads keep between calls: several threads
downloading from one batch, downloads without pinned memory, and the calls
that give the memory back."""
import math
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from ns3d_wcns_b200.config import GridDesc, make_params
from ns3d_wcns_b200.initial import isotropic_state, shock_tube_state

pytestmark = pytest.mark.gpu


def batch(sizes):
    from ns3d_wcns_b200.batch import Batch
    P, _ = make_params(n=(8, 4, 4), Ma=1.0, Re=math.inf, cfl=0.5, interpolation=0, riemann=0, bcs=(3, 3, 0, 0, 0, 0))
    b = Batch(P, [GridDesc(global_nx=n, global_ny=4, global_nz=4, Lx=1.0, Ly=1.0, Lz=1.0) for n in sizes], [0.2] * len(sizes))
    rng = np.random.default_rng(2)
    for i, n in enumerate(sizes):
        side = lambda: (rng.uniform(0.1, 1.0), rng.uniform(-1, 1), rng.uniform(0.1, 3.5))
        b.set_interior_primitives(i, *shock_tube_state(n, 4, 4, side(), side()))
    b.run(5)
    return b


def test_threads_download(gpu_lib):
    """Each thread gets its problem's state although they share the batch's pinned buffer."""
    sizes = [200, 1600, 400, 800] * 8
    with batch(sizes) as b, ThreadPoolExecutor(8) as pool:
        want = [b.primitives(i) for i in range(len(sizes))]
        for _ in range(4):
            for a, w in zip(pool.map(b.primitives, range(len(sizes))), want):
                assert np.array_equal(a, w)


def test_unpinned_download(gpu_lib):
    with batch([48, 200, 31]) as b:
        want = [b.primitives(i) for i in range(3)]
        assert b.lib.ns3d_debug_batch_unpinned(b.h) == 0
        for i in range(3):
            assert np.array_equal(b.primitives(i), want[i])


def test_release(gpu_lib):
    import torch
    from ns3d_wcns_b200.solver import Solver
    n = (40, 36, 32)
    P, G = make_params(n=n, Ma=0.3, Re=200.0, interpolation=0, riemann=0)
    rng = np.random.default_rng(3)
    with Solver(P, G) as s:
        s.set_interior_primitives(*isotropic_state(n, P.gamma, P.Ma, seed=11))
        ubar = rng.standard_normal((5,) + s.shape)
        s.compute_rhs()
        before = torch.cuda.mem_get_info()[0]
        first = s.adjoint_kinetic_energy(4, 1e-3, 2)[:2], s.vjp_rk3_step(1e-3, ubar), s.vjp_rhs(ubar)
        held = before - torch.cuda.mem_get_info()[0]
        s.release_scratch()
        # 69 interior arrays, and 2 checkpoints + 2 steps of 3 stages of 5 padded ones
        assert held >= 8 * (69 * n[0] * n[1] * n[2] + 40 * s.sx * s.sy * s.sz)
        assert before - torch.cuda.mem_get_info()[0] <= held // 8
        again = s.adjoint_kinetic_energy(4, 1e-3, 2)[:2], s.vjp_rk3_step(1e-3, ubar), s.vjp_rhs(ubar)
    assert first[0][0] == again[0][0] and np.array_equal(first[0][1], again[0][1])
    assert np.array_equal(first[1], again[1]) and np.array_equal(first[2], again[2])
    with batch([48, 200]) as b:
        want = b.primitives(1)
        b.release_scratch()
        assert np.array_equal(b.primitives(1), want)
