"""GPU: the ray cast's edge lists against the oracle, exactly: polygons of
fewer edges than a list pass holds, of exactly one and two passes and one more
or less, rows of cells that end inside a block, cells that hold many vertices,
and a body partly outside the grid."""
import numpy as np
import pytest

from ntustcfdlab_b200.abi import make_params

pytestmark = pytest.mark.gpu


def _blob(npts):
    """A closed, star-shaped outline of npts points (the last repeats the first), not symmetric."""
    t = 2.0 * np.pi * np.arange(npts - 1) / (npts - 1) + 0.0137
    r = 0.61 + 0.13 * np.sin(3 * t + 0.4) + 0.07 * np.cos(5 * t)
    z, y = 0.5 + r * np.cos(t), 0.8 * r * np.sin(t)
    return np.append(z, z[0]), np.append(y, y[0])


@pytest.mark.parametrize("npts", [4, 33, 128, 129, 130, 256, 257, 258, 514, 900])
@pytest.mark.parametrize("n,at", [((3, 24, 29), (2.0137, 1.5071)), ((4, 57, 131), (2.0137, 1.5071)),
                                  ((3, 40, 256), (3.7137, 2.6071))])
def test_polygon_mask_equals_oracle(orc, n, at, npts):
    from ntustcfdlab_b200.solver import Solver, gridder_equal
    g = gridder_equal(*n, 1.0, 3.0, 4.0)
    p = make_params(*n, Re=100.0, dt=1e-3)
    z, y = _blob(npts)
    with Solver(p, g) as s:
        assert s.build_mask_polygon(z, y, 7.3, *at) == 0
        eta = s.get_mask()
    o = orc.Oracle(p, g)
    assert o.raycasting(z, y, 7.3, *at) == 0
    np.testing.assert_array_equal(eta, o.get("ETA"))
    assert 0.0 < eta.sum()
