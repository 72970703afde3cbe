"""GPU: the marching SOR kernel (the solve of grids whose e does not fit the
chip) against the resident kernel, at the edges of its tiles: rows that just
fit and just miss a row pitch, odd and even rows, one tile and many, fewer
rows than a tile holds, ranges of one plane and of several, restarts, and a
stop test every few sweeps.

Both kernels sum a cell's terms in one order.  FP32 also rounds 1/diag to
nearest in both; in FP64 one forms it from the 1-D tables to within an ulp, so
a value differs by at most an ulp per sweep and the fields by 60 of them: the
repository's 1e-12 for two paths.  The last change is a difference of values
of order 1 and not below 1e-5 after 60 sweeps at most: 60 ulp of 1 in 1e-5,
about 1e-9.
"""
import numpy as np
import pytest

from conftest import interior, rel_l2
from ntustcfdlab_b200.abi import FP64, MIXED, SOR_AUTO, SOR_RESIDENT, SOR_STREAMING, f4, make_params

pytestmark = pytest.mark.gpu

SIZES = [(3, 3, 4), (46, 31, 40), (47, 61, 5), (78, 23, 17), (79, 5, 160), (142, 21, 9), (143, 14, 11), (234, 9, 12),
         (17, 200, 300), (64, 90, 96)]


def _solve(n, precision, path, reported, **kw):
    from ntustcfdlab_b200.solver import Solver, gridder_equal
    p = make_params(*n, Re=100.0, dt=f4(1e-3), precision=precision, sor_path=path,
                    bc={"North": ("Dirichlet", "no-slip", "no-slip")}, **kw)
    rng = np.random.default_rng(sum(n))
    shape = tuple(d + 4 for d in n)
    with Solver(p, gridder_equal(*n, 1.0, 1.1, 0.9)) as s:
        s.set_state(*[np.asfortranarray(0.3 * rng.standard_normal(shape)) for _ in range(4)])
        s.boundary_conditions()
        info, _ = s.step(2)
        assert {i.sor_path for i in info} == {reported}
        return s.get_state(), [(i.sor_iters, i.converged, i.dc_cycles) for i in info], [i.sor_last_change for i in info]


def _same(a, b):
    (x, ix, cx), (y, iy, cy) = a, b
    assert ix == iy
    assert np.allclose(cx, cy, rtol=1e-9, atol=0)
    for f, g in zip(x, y):
        assert rel_l2(interior(f), interior(g)) <= 1e-12


@pytest.mark.parametrize("precision", [FP64, MIXED])
@pytest.mark.parametrize("n", SIZES)
def test_march_equals_resident(n, precision):
    kw = dict(mixed_cycle=5, check_every=1 if n[0] % 2 else 5, itmax=60, zeta=1e-3)
    _same(_solve(n, precision, SOR_STREAMING, SOR_STREAMING, **kw), _solve(n, precision, SOR_RESIDENT, SOR_RESIDENT, **kw))


@pytest.mark.parametrize("precision,chosen", [(MIXED, SOR_STREAMING), (FP64, SOR_RESIDENT)])
def test_auto_takes_the_faster_kernel_and_keeps_the_result(precision, chosen):
    n, kw = (33, 150, 220), dict(itmax=24, zeta=0.0)
    _same(_solve(n, precision, SOR_AUTO, chosen, **kw), _solve(n, precision, SOR_RESIDENT, SOR_RESIDENT, **kw))
