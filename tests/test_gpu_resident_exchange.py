"""GPU: the resident SOR kernel's bricks and its exchange between CTAs against
the streaming kernels, at the edges of its row shapes: rows shorter than a
warp (several side by side), odd row lengths (the two colours differ by a
cell), one- and two-chunk rows, bricks of two rows, a grid that runs in one
CTA, correction cycles (restarts) and a stop test every few sweeps.

Both paths evaluate the same red-black sweeps with the same rounding, so the
fields agree to the repository's 1e-12 for two paths and the sweep counts
are equal.
"""
import numpy as np
import pytest

from conftest import interior, rel_l2
from ntustcfdlab_b200.abi import FP64, MIXED, SOR_RESIDENT, SOR_STREAMING, f4, make_params

pytestmark = pytest.mark.gpu

SIZES = [(3, 3, 3), (12, 10, 8), (5, 37, 6), (16, 24, 25), (33, 20, 18), (40, 40, 13), (63, 9, 31), (64, 30, 7),
         (65, 12, 29), (131, 8, 16), (257, 6, 5)]


def _solve(n, precision, path, **kw):
    from ntustcfdlab_b200.solver import Solver, gridder_equal
    p = make_params(*n, Re=100.0, dt=f4(1e-3), precision=precision, sor_path=path,
                    bc={"North": ("Dirichlet", "no-slip", "no-slip")}, **kw)
    rng = np.random.default_rng(sum(n))
    shape = tuple(d + 4 for d in n)
    with Solver(p, gridder_equal(*n, 1.0, 1.1, 0.9)) as s:
        s.set_state(*[np.asfortranarray(0.3 * rng.standard_normal(shape)) for _ in range(4)])
        s.boundary_conditions()
        info, _ = s.step(2)
        assert {i.sor_path for i in info} == {path}
        return s.get_state(), [(i.sor_iters, i.converged, i.dc_cycles) for i in info], [i.sor_last_change for i in info]


@pytest.mark.parametrize("precision", [FP64, MIXED])
@pytest.mark.parametrize("n", SIZES)
def test_resident_equals_streaming(n, precision):
    kw = dict(mixed_cycle=5, check_every=1 if n[0] % 2 else 5, itmax=60, zeta=1e-3)
    a, ia, ca = _solve(n, precision, SOR_RESIDENT, **kw)
    b, ib, cb = _solve(n, precision, SOR_STREAMING, **kw)
    assert ia == ib
    assert np.allclose(ca, cb, rtol=1e-6 if precision == MIXED else 1e-12, atol=0)
    for x, y in zip(a, b):
        assert rel_l2(interior(x), interior(y)) <= 1e-12
