"""The status word: kernels set its bits on the device and once in the host's copy, and a new
start clears both."""
import numpy as np
import pytest

from cppimpact_gb300 import meshgen as mg
from test_gpu_resident_limits import E, NU, RHO

pytestmark = pytest.mark.gpu

FORMS = [(1, 8, dict(step_kernel=3)), (1, 40, dict(step_kernel=3)), (1, 8, dict(step_kernel=1)),
         (2, 6, dict(step_kernel=3)), (2, 6, dict(step_kernel=2)), (2, 24, dict(step_kernel=3)),
         (2, 6, dict(step_kernel=3, elem_lanes=1)), (2, 6, dict(step_kernel=1))]


@pytest.mark.parametrize("order,n,kw", FORMS)
def test_bits_and_new_start(cilib, order, n, kw):
    """Every kernel that reports: a node whose velocity overflows FP32 (not finite), every element
    turned inside out (det J not positive), again after a new start, and none of it in a run
    without either."""
    m = mg.cube(n, order)
    setup = mg.impact_setup(m, 20.0, 1e-4)
    s = cilib.Solver(m.xloc, m.conn, E=E, nu=NU, rho=RHO, sigma_y0=100e6, H=0.689e9,
                     mode=cilib.MODE_J2, lumping=cilib.LUMP_HRZ, wall_normal=setup["wall_normal"],
                     wall_offset=setup["wall_offset"], wall_stiffness=setup["wall_stiffness"], **kw)
    for _ in range(2):
        s.initialize(setup["vel"])
        s.start(setup["dt"])
        assert s.status() == 0
        s.step(3)
        assert s.status() == 0
        s.set_state(m.xloc * [1.0, 1.0, -1.0], np.zeros((m.num_nodes, 3)))
        with pytest.raises(cilib.CiError) as e:
            s.step(2)
        assert e.value.code == -3 and s.status() & 1
        s.initialize(setup["vel"])
        s.start(setup["dt"])
        assert s.status() == 0
        v = np.zeros((m.num_nodes, 3))
        v[0] = 1e300
        s.set_state(m.xloc, v)
        with pytest.raises(cilib.CiError) as e:
            s.step(1)
        assert e.value.code in (-3, -4) and s.status() & 2
    s.close()
