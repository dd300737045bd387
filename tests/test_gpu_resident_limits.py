"""The resident step kernel's bounded waits: a chunk that never publishes its slots (test hook)
ends the call with an error, whatever else the run reports, and a solver that starts again
steps as a new one."""
import time

import numpy as np
import pytest

from cppimpact_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu

E, NU, RHO = 68.9e9, 0.33, 2700.0


def start(cilib, m, setup, s=None):
    s = s or cilib.Solver(m.xloc, m.conn, E=E, nu=NU, rho=RHO, sigma_y0=100e6, H=0.689e9,
                          mode=cilib.MODE_J2, lumping=cilib.LUMP_HRZ,
                          wall_normal=setup["wall_normal"], wall_offset=setup["wall_offset"],
                          wall_stiffness=setup["wall_stiffness"], step_kernel=3)
    s.initialize(setup["vel"])
    s.start(setup["dt"])
    return s


@pytest.mark.parametrize("order,n", [(1, 10), (2, 12)])
@pytest.mark.parametrize("nan", [False, True])
def test_resident_wait_gives_up(cilib, order, n, nan):
    """With a NaN velocity in every node the run has no positive det J either, and says so."""
    m = mg.cube(n, order)
    setup = mg.impact_setup(m, 20.0, 1e-4)
    s = start(cilib, m, setup)
    if nan:
        s.set_state(m.xloc, np.full((m.num_nodes, 3), np.nan))
    s.debug_flow_stall(1, 0.2)
    t0 = time.perf_counter()
    with pytest.raises(cilib.CiError) as e:
        s.step(50)
    assert e.value.code == (-3 if nan else -2)
    assert nan or "time limit" in str(e.value)
    assert s.status() & 8 and time.perf_counter() - t0 < 30.0
    with pytest.raises(cilib.CiError):   # until it starts again
        s.step(1)
    start(cilib, m, setup, s)
    assert s.status() == 0
    fresh = start(cilib, m, setup)
    for k in (1, 60):
        s.step(k)
        fresh.step(k)
    a, b = s.state(), fresh.state()
    for k in a:
        assert np.array_equal(a[k], b[k]), k
    assert not np.array_equal(a["x"], m.xloc)
    s.close()
    fresh.close()
