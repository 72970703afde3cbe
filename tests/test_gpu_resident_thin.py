"""GPU: grids of long rows that fit the chip only in bricks of one row (a row
then goes to up to four neighbours) or just fit it in bricks of two, on the
resident SOR kernel against the streaming path.

Both evaluate the same sweeps in one order of operations, so the sweep counts
are equal; the fields are held to the repository's 1e-12 for two paths (40 sweeps of
at most an ulp), the last change to 40 ulp of 1 in 1e-5 or more: 1e-9.
"""
import numpy as np
import pytest

from conftest import interior, rel_l2
from ntustcfdlab_b200.abi import FP64, MIXED, SOR_RESIDENT, SOR_STREAMING, f4, make_params

pytestmark = pytest.mark.gpu

CASES = [(FP64, n) for n in [(1572, 6, 3), (1210, 27, 7), (1567, 97, 3), (1800, 3, 70), (2218, 11, 5), (2317, 14, 10),
                             (1386, 21, 20), (1059, 37, 13), (89, 256, 118)]]
CASES += [(MIXED, n) for n in [(2128, 11, 5), (3351, 38, 3), (2672, 18, 29), (3317, 29, 5), (2478, 3, 235),
                               (51, 509, 217), (522, 26, 349)]]


def _solve(n, precision, path, **kw):
    from ntustcfdlab_b200.solver import Solver, gridder_equal
    p = make_params(*n, Re=100.0, dt=f4(1e-3), precision=precision, sor_path=path,
                    bc={"North": ("Dirichlet", "no-slip", "no-slip")}, **kw)
    rng = np.random.default_rng(sum(n))
    shape = tuple(d + 4 for d in n)
    with Solver(p, gridder_equal(*n, n[0] / 40, 1.1, 0.9)) as s:
        s.set_state(*[np.asfortranarray(0.3 * rng.standard_normal(shape)) for _ in range(4)])
        s.boundary_conditions()
        info, _ = s.step(2)
        assert {i.sor_path for i in info} == {path}
        return s.get_state(), [(i.sor_iters, i.converged, i.dc_cycles) for i in info], [i.sor_last_change for i in info]


@pytest.mark.parametrize("precision,n", CASES)
def test_long_rows_fit_and_equal_streaming(precision, n):
    kw = dict(mixed_cycle=7, check_every=1, itmax=40, zeta=1e-3)
    a, ia, ca = _solve(n, precision, SOR_RESIDENT, **kw)
    b, ib, cb = _solve(n, precision, SOR_STREAMING, **kw)
    assert ia == ib
    assert np.allclose(ca, cb, rtol=1e-9, atol=0)
    for x, y in zip(a, b):
        assert rel_l2(interior(x), interior(y)) <= 1e-12
