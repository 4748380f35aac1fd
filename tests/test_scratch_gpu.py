"""Batch downloads: several threads at once, and without pinned memory."""
import math
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from ns3d_wcns_b200.config import GridDesc, make_params
from ns3d_wcns_b200.initial import shock_tube_state

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
