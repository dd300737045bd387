"""State read into page-locked, pageable and partly page-locked arrays, on both sides of the
size up to which the kernel writes page-locked arrays itself."""
import numpy as np
import pytest

from cppimpact_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 19, 20])
def test_same_values(cilib, n):
    """Cubes of 27, 8,000 and 9,261 nodes: the same bits in whatever memory; the entries
    beside the arrays stay."""
    torch = pytest.importorskip("torch")
    m = mg.cube(n, 1)
    setup = mg.impact_setup(m, 20.0, 0.0)
    s = cilib.Solver(m.xloc, m.conn, E=68.9e9, nu=0.33, rho=2700.0, sigma_y0=276e6, H=0.689e9,
                     wall_normal=setup["wall_normal"],
                     wall_offset=setup["wall_offset"], wall_stiffness=setup["wall_stiffness"])
    s.initialize(setup["vel"])
    s.start(setup["dt"])
    s.step(3)
    x, v = np.empty((m.num_nodes, 3)), np.empty((m.num_nodes, 3))
    s.get_xv(x, v)
    assert np.isfinite(x).all() and np.isfinite(v).all()
    size = 3 * m.num_nodes
    pinned = torch.full((2 * size + 3,), 7.0, dtype=torch.float64, pin_memory=True).numpy()
    px, pv = pinned[1:1 + size], pinned[2 + size:2 + 2 * size]
    s.get_xv(px, pv)
    assert np.array_equal(px, x.ravel()) and np.array_equal(pv, v.ravel())
    assert (pinned[[0, 1 + size, -1]] == 7.0).all()
    pv[:] = 0.0
    x2 = np.empty_like(x)
    s.get_xv(x2, pv)  # one of each
    assert np.array_equal(x2, x) and np.array_equal(pv, v.ravel())
    s.close()
