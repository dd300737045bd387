"""The fused step held on the GPU for all steps of a call against a launch per step, on the same
plan and with the form of either asserted: states, accelerations and work sums to the bit."""
import numpy as np
import pytest

from cppimpact_gb300 import meshgen as mg
from test_gpu_shared_limits import solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,n,threads", [(1, 3, 128), (1, 10, 128), (1, 14, 64), (1, 15, 128),
                                             (1, 30, 128), (1, 10, 256), (2, 4, 128), (2, 13, 128),
                                             (2, 18, 128)])
@pytest.mark.parametrize("mode", ["j2", "refcompat"])
def test_resident_equals_launches(cilib, order, n, threads, mode):
    """tet4 chunks of at most 32 elements (CTAs of 64 threads) and more, tet10 up to 58; calls of
    one and of many steps through a yielding contact."""
    m = mg.cube(n, order)
    setup = mg.impact_setup(m, 30.0, 1e-5)
    out = []
    for use in (1, 0):
        s = solver(cilib, m, setup, step_kernel=3, block_threads=threads)
        if mode == "refcompat":
            s.close()
            s = cilib.Solver(m.xloc, m.conn, E=68.9e9, nu=0.33, rho=2700.0,
                             mode=cilib.MODE_REFCOMPAT, lumping=cilib.LUMP_HRZ,
                             wall_normal=setup["wall_normal"], wall_offset=setup["wall_offset"],
                             wall_stiffness=setup["wall_stiffness"], step_kernel=3,
                             block_threads=threads)
            s.initialize(setup["vel"])
            s.start(setup["dt"])
        assert s.debug_resident(use) == bool(use)
        for k in (1, 2, 41, 60):
            s.step(k)
        assert s.debug_resident() == bool(use)
        out.append((s.state(), s.nodal_fields()["acc"], s.energy()))
        s.close()
    (a, acc_a, ea), (b, acc_b, eb) = out
    assert (a["contact"] & 2).any()
    for k in a:
        assert np.array_equal(a[k], b[k]), k
    assert np.array_equal(acc_a, acc_b)
    assert ea["internal"] == eb["internal"] and ea["plastic"] == eb["plastic"]


def test_forms_in_turn(cilib):
    """One solver that changes its form between calls steps as one that does not."""
    m = mg.cube(10, 1)
    setup = mg.impact_setup(m, 30.0, 1e-5)
    out = []
    for turns in ((1, 1, 1, 1), (0, 1, 0, 1)):
        s = solver(cilib, m, setup)
        for use, k in zip(turns, (7, 20, 1, 32)):
            assert s.debug_resident(use) == bool(use)
            s.step(k)
        out.append(s.state())
        s.close()
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k


def test_larger_plans_launch(cilib):
    """Chunks that do not fit, and every solver but the fused one's."""
    m = mg.cube(24, 2)
    setup = mg.impact_setup(m, 30.0, 1e-5)
    for kw in (dict(step_kernel=3), dict(step_kernel=1), dict(step_kernel=2), dict(elem_lanes=1)):
        s = solver(cilib, m, setup, **kw)
        assert not s.debug_resident(1)
        s.close()
