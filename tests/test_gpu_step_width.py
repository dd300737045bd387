"""The step kernels' widths (CTAs wider than block_threads): on one plan the state does not
depend on them."""
import numpy as np
import pytest

from cppimpact_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu

E, NU, RHO = 68.9e9, 0.33, 2700.0


def solve(cilib, m, mode, **shape):
    setup = mg.impact_setup(m, 30.0, 1e-5)
    s = cilib.Solver(m.xloc, m.conn, E=E, nu=NU, rho=RHO, sigma_y0=100e6, H=0.689e9,
                     mode=cilib.MODE_J2 if mode == "j2" else cilib.MODE_REFCOMPAT,
                     lumping=cilib.LUMP_HRZ, wall_normal=setup["wall_normal"],
                     wall_offset=setup["wall_offset"], wall_stiffness=setup["wall_stiffness"],
                     step_kernel=3, **shape)
    s.initialize(setup["vel"])
    s.start(setup["dt"])
    for k in (1, 2, 41, 60):
        s.step(k)
    out = s.state(), s.energy()
    s.close()
    return out


@pytest.mark.parametrize("n,elements,nodes,mode", [(16, 520, 512, "j2"), (20, 1030, 512, "j2"),
                                                   (24, 2048, 896, "refcompat"),
                                                   (16, 4096, 1500, "j2"), (40, 0, 896, "j2")])
def test_state_and_work(cilib, n, elements, nodes, mode):
    """Chunks of a little over and under two, four and eight windows: states equal bit for
    bit for blocks of 64, 128 and 256 threads (four, two and one window at a time), the work
    sums (FP32 within a chunk and step, in an order of the block size) to 1e-5."""
    m = mg.cube(n, 1)
    out = [solve(cilib, m, mode, chunk_elements=elements, chunk_nodes=nodes, block_threads=bs)
           for bs in (64, 128, 256)]
    a, ea = out[0]
    assert (a["contact"] & 2).any()
    for b, eb in out[1:]:
        for k in ("x", "v", "sigma", "epbar", "contact"):
            assert np.array_equal(a[k], b[k]), k
        for k in ("internal", "plastic"):
            assert eb[k] == pytest.approx(ea[k], rel=1e-5), k


@pytest.mark.parametrize("n,elements,nodes,mode", [(12, 300, 896, "j2"), (17, 97, 512, "refcompat"),
                                                   (20, 250, 896, "j2"), (22, 150, 896, "j2"),
                                                   (20, 0, 896, "refcompat")])
def test_state_and_work_tet10(cilib, n, elements, nodes, mode):
    """The four-lane kernel with 384, 256 and 192 threads for the 128 asked for (35 to 608
    chunks) against 64 and 256: states equal bit for bit, work sums as above."""
    m = mg.cube(n, 2)
    out = [solve(cilib, m, mode, chunk_elements=elements, chunk_nodes=nodes, block_threads=bs)
           for bs in (64, 128, 256)]
    a, ea = out[0]
    for b, eb in out[1:]:
        for k in ("x", "v", "sigma", "epbar", "contact"):
            assert np.array_equal(a[k], b[k]), k
        for k in ("internal", "plastic"):
            assert eb[k] == pytest.approx(ea[k], rel=1e-5), k


def test_repeated_node(cilib):
    """A tet10 that names a corner as one of its own edge nodes (its Jacobian stays positive at
    the Gauss points) steps on the one-lane kernel, whatever kernel was asked for."""
    m = mg.cube(20, 2)
    m.conn[7, 4] = m.conn[7, 0]
    out = [solve(cilib, m, "j2", chunk_elements=700, **k)[0]
           for k in (dict(elem_lanes=1), dict(elem_lanes=4))]
    for k in ("x", "v", "sigma", "epbar", "contact"):
        assert np.array_equal(out[0][k], out[1][k]), k
