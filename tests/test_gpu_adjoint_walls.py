"""GPU: the transposed boundary conditions on the shortest lines (three cells,
where the second cell from one wall is the first from the other) and the next
longer ones, for each kind of wall along x, against central differences of
complete runs, to the tolerance of the other gradient tests."""
import numpy as np
import pytest

from ntustcfdlab_b200 import abi, cases
from test_gpu_adjoint import FD_RTOL, K, _fd, initial_state, objective, run_adjoint

pytestmark = pytest.mark.gpu


def _case(nx, kind, U=1.0):
    c = cases.cylinder_crossflow(nx, 24, 32, 1.0, 6.0, 8.0, zc=2.55, yc=3.1, D=1.0, Re=100.0, dt=0.01, U=U,
                                 theta_deg=5.0, steps=K, precision=abi.FP64, zeta=1e-12, itmax=200000)
    for wall in (0, 1):
        for comp in range(3):
            c.params.bc[wall][comp] = kind
    return c


@pytest.mark.parametrize("nx", [3, 4, 5])
@pytest.mark.parametrize("kind", [0, 1, 2, 3], ids=["no-slip", "neumann", "dirichlet", "periodic"])
def test_short_lines_match_central_differences(nx, kind):
    case = _case(nx, kind)
    state = initial_state(case)
    force = cases.body_force_c4((nx, 24, 32), scale=1e-2)
    r = run_adjoint(case, state, force)
    gU = _fd(lambda U: objective(_case(nx, kind, U), state, force), 1.0)
    assert abs(r["dJ_dU"] - gU) <= FD_RTOL * abs(gU), (r["dJ_dU"], gU)
