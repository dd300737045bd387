"""The task kernel with element and node tasks in turns (long meshes of many chunks)."""
import numpy as np
import pytest

from cppimpact_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu

E, NU, RHO = 68.9e9, 0.33, 2700.0


@pytest.mark.parametrize("around,axial,elements,steps", [(24, 700, 64, (1, 2, 5)),
                                                         (24, 500, 64, (3, 1, 4)),
                                                         (48, 500, 100, (7,))])
def test_equals_a_launch_per_step(cilib, around, axial, elements, steps):
    """Enough chunks for turns (about 1,600 and 1,440 of 24 to 48 cells around; 1,125 at the
    edge) against the fused kernel on the same plan: the same bits."""
    m = mg.shell(around, axial, order=2)
    setup = mg.impact_setup(m, 30.0, 0.0)
    out = []
    for kernel in (2, 3):
        s = cilib.Solver(m.xloc, m.conn, E=E, nu=NU, rho=RHO, sigma_y0=100e6, H=0.689e9,
                         wall_normal=setup["wall_normal"], wall_offset=setup["wall_offset"],
                         wall_stiffness=setup["wall_stiffness"], step_kernel=kernel,
                         chunk_elements=elements, chunk_nodes=512)
        assert s.step_kernel() == kernel
        s.initialize(setup["vel"])
        s.start(setup["dt"])
        for k in steps:
            s.step(k)
        out.append(s.state())
        s.close()
    for k in ("x", "v", "sigma", "epbar", "contact"):
        assert np.array_equal(out[0][k], out[1][k]), k
