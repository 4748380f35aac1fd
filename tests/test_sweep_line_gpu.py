"""The x-sweep (a line per warp, two faces per lane, chunks of 64 faces) where
it can go wrong: lines that end just before, at and after a chunk, the
shortest ones, line counts that leave warps idle, odd and even line pairs, and
every boundary type, against the CPU oracle.  Tolerance: the FP64 path's own
bounds, 1e-12 of the largest right-hand side and 1e-10 of the state after two
steps.  Mixed path (continuous schemes): two steps change the state by less
than a tenth, in FP32 to some 1e-6 of that, so 1e-6 of the state."""
import pytest

from helpers import interior, rel_linf
from ns3d_wcns_b200.config import make_params
from ns3d_wcns_b200.initial import random_state
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(61, 5, 60), (61, 60, 3), (55, 67, 7), (66, 62, 64)], ids=str)
@pytest.mark.parametrize("bcs", [(0,) * 6, (3, 3, 1, 2, 4, 4), (1, 2, 3, 3, 0, 0)],
                         ids=["periodic", "mixed", "z-periodic"])
@pytest.mark.parametrize("interp,rs", [(0, 0), (3, 2), (2, 2)])
def test_many_lines_against_oracle(gpu_lib, n, bcs, interp, rs):
    """More lines than the kernel with a line per warp takes along y and z:
    the marching kernel, whole lines and segments."""
    _check(n, bcs, interp, rs)

NX = [3, 4, 58, 59, 60, 61, 63, 64, 65, 66, 124, 128, 131]
BCS = [(0,) * 6, (3, 3, 0, 0, 1, 2), (1, 2, 3, 3, 0, 0)]


@pytest.mark.parametrize("nx", NX)
@pytest.mark.parametrize("ny", [4, 5])
@pytest.mark.parametrize("bcs", BCS, ids=["periodic", "outflow", "wall"])
@pytest.mark.parametrize("interp,rs", [(0, 0), (3, 2), (2, 2)])
def test_sweep_line_against_oracle(gpu_lib, nx, ny, bcs, interp, rs):
    _check((nx, ny, 3), bcs, interp, rs)


def _check(n, bcs, interp, rs):
    from ns3d_wcns_b200.solver import Solver
    P, G = make_params(n=n, L=(1.0, 0.8, 0.9), interpolation=interp, riemann=rs, bcs=bcs, Re=300.0, dt_fixed=1e-4)
    st = random_state(n, seed=7, amp=0.2)
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
    if interp == 3:  # its detector may flip at a threshold in FP32
        return
    Pm, _ = make_params(n=n, L=(1.0, 0.8, 0.9), interpolation=interp, riemann=rs, bcs=bcs, Re=300.0, dt_fixed=1e-4,
                        precision=1)
    with Solver(Pm, G) as s:
        s.set_interior_primitives(*st)
        for _ in range(2):
            s.rk3_step(1e-4)
        for a, b in zip(interior(s.conserved()), interior(o.conserved())):
            assert rel_linf(a, b) <= 1e-6


@pytest.mark.parametrize("n", [(592, 3, 3), (122, 16, 16), (122, 14, 4)], ids=str)
@pytest.mark.parametrize("char_recon", [0, 1])
def test_stage_partials(gpu_lib, n, char_recon):
    """The time step and the kinetic energy come from the partials that the
    z-sweep's blocks leave: more blocks than the padded grid has rows of 128.
    Tolerance: the state's 1e-10."""
    from ns3d_wcns_b200.solver import Solver
    P, G = make_params(n=n, L=(6.0, 0.8, 0.9), interpolation=2, riemann=2, Re=300.0, cfl=0.4, char_recon=char_recon)
    st = random_state(n, seed=9, amp=0.2)
    o = oracle.PortSolver(P, G)
    o.set_interior_prims(*st)
    with Solver(P, G) as s:
        s.set_interior_primitives(*st)
        for _ in range(3):
            dt = o.timestep()
            assert abs(s.compute_timestep() / dt - 1) <= 1e-10
            s.rk3_step(dt)
            o.rk3_step(dt)
        W = [interior(o.get(k)) for k in ("rho", "u", "v", "w")]
        dv = 6.0 / n[0] * 0.8 / n[1] * 0.9 / n[2]
        ke = float((0.5 * W[0] * (W[1] ** 2 + W[2] ** 2 + W[3] ** 2)).sum() * dv)
        assert abs(s.total_energy() / ke - 1) <= 1e-10


@pytest.mark.parametrize("n", [(60, 61, 5), (64, 5, 62), (5, 63, 64), (62, 64, 60)], ids=str)
@pytest.mark.parametrize("bcs", [(0,) * 6, (0, 0, 0, 0, 1, 3), (3, 2, 0, 0, 0, 0)], ids=["periodic", "xy", "yz"])
@pytest.mark.parametrize("interp,rs", [(0, 0), (3, 2)])
def test_one_chunk_lines(gpu_lib, n, bcs, interp, rs):
    """Periodic lines of 60 to 64 cells take one chunk whose first positions
    update the line's last cells."""
    _check(n, bcs, interp, rs)
