"""GPU: a context whose pressure solves march holds one set of colour arrays,
and holds it from its creation on, so that the choice of the kernel rests on
the grid and the device and not on the memory that happens to be free at a
later step; the z-slab stages of such a context make the colour-split ones."""
import numpy as np
import pytest

from ntustcfdlab_b200 import abi
from ntustcfdlab_b200.abi import FP64, MIXED, SOR_STREAMING, f4, make_params

pytestmark = pytest.mark.gpu

N = (128, 192, 256)
SLACK = 64 << 20        # kernels loaded, tables, records, faces, rounding of the allocations


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _solver(n, precision):
    from ntustcfdlab_b200.solver import Solver, gridder_equal
    p = make_params(*n, Re=100.0, dt=f4(1e-3), precision=precision, sor_path=SOR_STREAMING, itmax=4, zeta=0.0,
                    bc={"North": ("Dirichlet", "no-slip", "no-slip")})
    return Solver(p, gridder_equal(*n, 1.0, 1.1, 0.9))


@pytest.mark.parametrize("precision", [FP64, MIXED])
def test_colour_arrays_are_held_once_and_from_the_start(precision):
    with _solver((20, 16, 12), precision) as s:      # the kernels' own memory
        s.boundary_conditions()
        s.step(1)
    word = 8 if precision == FP64 else 4
    halo = (N[0] + 16) * (N[1] + 12) * (N[2] + 4)
    cells = N[0] * N[1] * N[2]
    before = _free()
    with _solver(N, precision) as s:
        made = before - _free()
        s.boundary_conditions()
        s.step(2)
        ran = before - _free()
        # nine natural arrays, the output, the force's columns, six colour arrays of half a halo each
        assert made <= 9 * 8 * halo + 4 * 8 * cells + 3 * word * halo + SLACK
        assert ran - made <= SLACK


def test_slab_stages_of_a_marching_context():
    n = (20, 16, 12)
    rng = np.random.default_rng(3)
    state = [np.asfortranarray(0.2 * rng.standard_normal(tuple(d + 4 for d in n))) for _ in range(4)]
    with _solver(n, FP64) as a, _solver(n, FP64) as b:
        for s in (a, b):
            s.set_state(*state)
            s.boundary_conditions()
        a.step(2)
        b.step(1)
        stage = lambda k, colour=0: b._check(b.lib.ntcfd_slab_stage(b.h, k, colour))
        stage(abi.STAGE_PREDICT)
        stage(abi.STAGE_RHS)
        for _ in range(4):
            stage(abi.STAGE_HALFSWEEP, 0)
            stage(abi.STAGE_HALFSWEEP, 1)
        stage(abi.STAGE_CORRECT)
        stage(abi.STAGE_PROJECT)
        for x, y in zip(a.get_state(), b.get_state()):
            # the same four sweeps, to the tolerance of two paths
            assert np.abs(x - y).max() <= 1e-12 * max(1.0, np.abs(x).max())
        b.boundary_conditions()
        b.step(1)


def test_velocity_planes_make_no_colour_arrays():
    with _solver(N, FP64) as s:
        s.boundary_conditions()
        s.step(1)
        n = s.lib.ntcfd_slab_plane_elems(s.h, abi.FIELD_U)
        buf = np.zeros(n)
        before = _free()
        s._check(s.lib.ntcfd_slab_planes(s.h, abi.FIELD_U, 1, 1, buf.ctypes.data, 0))
        assert before - _free() < 16 << 20
        s._check(s.lib.ntcfd_slab_planes(s.h, abi.FIELD_E_RED, 1, 1, buf.ctypes.data, 0))
        assert before - _free() > 6 * 8 * N[0] // 2 * N[1] * N[2]
