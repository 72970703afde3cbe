"""GPU: the resident kernel's form with a two-row ring (one hand-over a sweep,
the stop test judged a sweep late) against the streaming path: thin and thick
bricks, bricks cut along one direction only, rows of one to five side by side,
solves that end in the middle of a correction cycle, on its last sweep and on
the sweep limit, and a stop test every few sweeps.

Both evaluate the same sweeps in one order of operations, so the sweep counts
are equal; 1/diag may differ by an ulp in FP64, hence the repository's 1e-12
for two paths (60 ulp), and 60 ulp of 1 in a last change of 1e-5 or more: 1e-9.
"""
import numpy as np
import pytest

from conftest import interior, rel_l2
from ntustcfdlab_b200.abi import FP64, MIXED, SOR_RESIDENT, SOR_STREAMING, f4, make_params

pytestmark = pytest.mark.gpu

SIZES = [(6, 4, 3), (12, 10, 8), (5, 2 * 37, 3), (7, 3, 80), (13, 31, 33), (22, 24, 25), (33, 47, 29), (64, 40, 36)]


def _solve(n, precision, path, **kw):
    from ntustcfdlab_b200.solver import Solver, gridder_equal
    p = make_params(*n, Re=100.0, dt=f4(1e-3), precision=precision, sor_path=path,
                    bc={"North": ("Dirichlet", "no-slip", "no-slip")}, **kw)
    rng = np.random.default_rng(sum(n))
    shape = tuple(d + 4 for d in n)
    with Solver(p, gridder_equal(*n, 1.0, 1.1, 0.9)) as s:
        s.set_state(*[np.asfortranarray(0.3 * rng.standard_normal(shape)) for _ in range(4)])
        s.boundary_conditions()
        info, _ = s.step(3)
        assert {i.sor_path for i in info} == {path}
        return s.get_state(), [(i.sor_iters, i.converged, i.dc_cycles) for i in info], [i.sor_last_change for i in info]


@pytest.mark.parametrize("precision", [FP64, MIXED])
@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("zeta,itmax,cycle,every", [(1e-3, 60, 8, 1), (3e-2, 60, 5, 1), (1e-2, 60, 6, 3), (0.0, 11, 4, 1)])
def test_deep_ring_equals_streaming(n, precision, zeta, itmax, cycle, every):
    kw = dict(zeta=zeta, itmax=itmax, mixed_cycle=cycle, check_every=every)
    a, ia, ca = _solve(n, precision, SOR_RESIDENT, **kw)
    b, ib, cb = _solve(n, precision, SOR_STREAMING, **kw)
    assert ia == ib
    assert np.allclose(ca, cb, rtol=1e-9, atol=0)
    for x, y in zip(a, b):
        assert rel_l2(interior(x), interior(y)) <= 1e-12
