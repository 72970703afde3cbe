"""GPU: where the marching kernel looks at the stop rule in solves of several
correction cycles: every check_every sweeps of a cycle and at its end, as the
half-sweep loops do.  An adjoint solve with a higher sweep limit than the
context's runs FP64 cycles of the context's limit; with cycles of ten sweeps
and a test every four it can end on the fourth, eighth or tenth sweep of one."""
import numpy as np
import pytest

from ntustcfdlab_b200 import abi, cases
from ntustcfdlab_b200.solver import Solver

pytestmark = pytest.mark.gpu


def test_adjoint_solves_end_where_a_cycle_is_tested():
    c = cases.cylinder_crossflow(8, 24, 32, 1.0, 6.0, 8.0, zc=2.55, yc=3.1, D=1.0, Re=100.0, dt=0.01, U=1.0, theta_deg=5.0,
                                 steps=1, precision=abi.FP64, itmax=10, check_every=4, sor_path=abi.SOR_STREAMING)
    rng = np.random.default_rng(3)
    ends = set()
    with Solver(c.params, c.grid) as s:
        assert s.solve_plan()["kernel"] == abi.SOLVE_MARCH
        s.build_mask_cylinder(2.55, 3.1, 0.5)
        state = [np.asfortranarray(0.1 * rng.standard_normal(s.halo_shape)) for _ in range(3)]
        state.append(np.zeros(s.halo_shape, order="F"))
        state[2] += 1.0
        for zeta in (1e-1, 3e-2, 1e-2, 3e-3, 1e-3, 3e-4, 1e-4, 1e-5):
            s.set_state(*state)
            s.boundary_conditions()
            r = s.adjoint(1, 1, w_drag=1.0, adj_zeta=zeta, adj_itmax=4000, inflow=("Back", 2, 1))
            assert r["adj_unconverged"] == 0
            ends.add(r["adj_sweeps"] % 10)
    assert ends <= {0, 4, 8}, ends
