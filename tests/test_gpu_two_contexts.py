"""GPU: two contexts whose pressure solves run in the same kernel with shared
memory of different sizes.  The second one's smaller need leaves the first
one's launches as they were, in eager steps and in adjoint solves."""
import numpy as np
import pytest

from ntustcfdlab_b200.abi import FP64, MIXED, SOR_RESIDENT, SOR_STREAMING, f4, make_params

pytestmark = pytest.mark.gpu

# (large, small) grids that take one instance: two-row ring, one-row ring, marching, long rows
PAIRS = [(SOR_RESIDENT, (40, 40, 40), (12, 10, 8)), (SOR_RESIDENT, (100, 100, 90), (100, 40, 30)),
         (SOR_STREAMING, (40, 96, 60), (34, 9, 8)), (SOR_RESIDENT, (300, 24, 24), (280, 5, 6))]


def _solver(n, precision, path, **kw):
    from ntustcfdlab_b200.solver import Solver, gridder_equal
    p = make_params(*n, Re=100.0, dt=f4(1e-3), precision=precision, sor_path=path, itmax=9, zeta=0.0,
                    bc={"North": ("Dirichlet", "no-slip", "no-slip")}, **kw)
    s = Solver(p, gridder_equal(*n, 1.0, 1.1, 0.9))
    s.boundary_conditions()
    return s


@pytest.mark.parametrize("precision", [FP64, MIXED])
@pytest.mark.parametrize("path,large,small", PAIRS)
def test_a_smaller_context_leaves_the_larger_one_alone(path, large, small, precision):
    with _solver(large, precision, path, eager=1) as a, _solver(large, precision, path) as alone:
        a.step(1)
        alone.step(2)
        with _solver(small, precision, path) as b:
            b.step(1)
            info, _ = a.step(1)
            assert info[0].sor_iters == 9
            for x, y in zip(a.get_state(), alone.get_state()):
                np.testing.assert_array_equal(x, y)
            a.build_mask_cylinder(0.45, 0.55, 0.2)
            r = a.adjoint(2, 1, w_drag=1.0, inflow=("Back", 2, 1))
            assert np.isfinite(r["J"]) and r["adj_sweeps"] > 0
