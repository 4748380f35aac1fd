"""z-slabs against the single domain, bit for bit, on grids where the two take
different kernels for the same lines: the domain's lines along y (the first
size of each path) or along z (the second) march, a slab's run a line per
warp (line_takes in sweep_line.cuh decides by the number of lines)."""
import numpy as np
import pytest

from helpers import interior
from ns3d_wcns_b200.config import make_params
from ns3d_wcns_b200.initial import random_state

pytestmark = pytest.mark.gpu

SCHEMES = [(0, 0), (0, 2), (0, 3), (2, 2), (2, 5), (3, 2), (3, 0), (3, 4)]  # interpolation, riemann
CASES = [((64, 48, 76), 0), ((40, 40, 76), 0), ((96, 48, 80), 1), ((48, 40, 76), 1), ((81, 48, 76), 1), ((41, 40, 76), 1)]


@pytest.mark.parametrize("n,precision", CASES, ids=str)
@pytest.mark.parametrize("scheme", SCHEMES, ids=str)
@pytest.mark.parametrize("bcs", [(0,) * 6, (3, 3, 1, 2, 3, 2)], ids=["periodic", "bounded"])
def test_slabs_equal_domain(gpu_lib, n, precision, scheme, bcs):
    from ns3d_wcns_b200.slab import InProcessSlabs
    from ns3d_wcns_b200.solver import Solver
    P, G = make_params(n=n, L=tuple(0.1 * m for m in n), interpolation=scheme[0], riemann=scheme[1], Re=300.0, bcs=bcs,
                       precision=precision)
    W = random_state(n, seed=5, amp=0.2)
    with Solver(P, G) as s, InProcessSlabs(P, G, 2) as slabs:
        s.set_interior_primitives(*W)
        slabs.set_interior_primitives(*W)
        for _ in range(2):
            s.rk3_step(1e-3)
            slabs.rk3_step(1e-3)
        a = interior(s.primitives())
        b = slabs.owned_primitives()[:, :, 3:-3, 3:-3]
    assert np.array_equal(a, b)


@pytest.mark.parametrize("bcs", [(0,) * 6, (3, 3, 1, 2, 3, 2)], ids=["periodic", "bounded"])
def test_mixed_pointers_stay(gpu_lib, bcs):
    """On the mixed path a caller may take the pointers once: the halos of every stage written through them."""
    from ns3d_wcns_b200 import _lib
    from ns3d_wcns_b200.slab import InProcessSlabs
    from ns3d_wcns_b200.solver import Solver
    n = (24, 20, 38)
    P, G = make_params(n=n, L=tuple(0.1 * m for m in n), interpolation=2, riemann=2, Re=300.0, bcs=bcs, precision=1)
    W = random_state(n, seed=5, amp=0.2)
    with Solver(P, G) as s, InProcessSlabs(P, G, 2) as slabs:
        s.set_interior_primitives(*W)
        slabs.set_interior_primitives(*W)
        kept = {}

        def planes(x, side, k0, count):
            from ns3d_wcns_b200.slab import device_planes
            key = (id(x), k0)
            if key not in kept:
                kept[key] = device_planes(x.s, k0, count)
            return kept[key]
        for x in slabs.slabs:
            x.planes = lambda side, k0, count, x=x: planes(x, side, k0, count)
        first = [x.s.device_fields(_lib.NS3D_PRIMITIVE)[0] for x in slabs.slabs]
        for _ in range(2):
            s.rk3_step(1e-3)
            for stage in (1, 2, 3):
                for x in slabs.slabs:
                    assert x.s.lib.ns3d_rk3_stage(x.s.h, stage, 1e-3) == 0
                assert [x.s.device_fields(_lib.NS3D_PRIMITIVE)[0] for x in slabs.slabs] == first
                slabs.exchange_halos()
        assert np.array_equal(interior(s.primitives()), slabs.owned_primitives()[:, :, 3:-3, 3:-3])
