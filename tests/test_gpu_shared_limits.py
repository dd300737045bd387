"""Solvers and batches of different chunk sizes in one process: a kernel's shared-memory limit is
the process's, so the next solver's must not be too small for the one before."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT
from cppimpact_gb300 import meshgen as mg
from test_gpu_resident_limits import E, NU, RHO

pytestmark = pytest.mark.gpu

LARGE = dict(chunk_nodes=1400, chunk_elements=4096)   # 56 KB of node records
SMALL = dict(chunk_nodes=300, chunk_elements=60)


def solver(cilib, m, setup, **kw):
    s = cilib.Solver(m.xloc, m.conn, E=E, nu=NU, rho=RHO, sigma_y0=100e6, H=0.689e9,
                     mode=cilib.MODE_J2, lumping=cilib.LUMP_HRZ, wall_normal=setup["wall_normal"],
                     wall_offset=setup["wall_offset"], wall_stiffness=setup["wall_stiffness"], **kw)
    s.initialize(setup["vel"])
    s.start(setup["dt"])
    return s


@pytest.mark.parametrize("order,kw", [(1, dict(step_kernel=1)), (1, dict(step_kernel=3)),
                                      (2, dict(step_kernel=1)), (2, dict(step_kernel=2)),
                                      (2, dict(step_kernel=3)), (2, dict(step_kernel=3, elem_lanes=1))])
def test_a_smaller_solver_comes_second(cilib, order, kw):
    m = mg.cube(16 if order == 1 else 10, order)
    setup = mg.impact_setup(m, 30.0, 1e-5)
    out = []
    for second in (False, True):
        s = solver(cilib, m, setup, **LARGE, **kw)
        t = solver(cilib, m, setup, **SMALL, **kw) if second else None
        s.step(40)
        s.start(setup["dt"])   # the mass once more
        s.step(40)
        out.append(s.state())
        s.close()
        if t:
            t.step(1)
            t.close()
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k


@pytest.mark.parametrize("order", [1, 2])
def test_a_smaller_batch_comes_second(cilib, order):
    m = mg.cube(16 if order == 1 else 10, order)
    setup = mg.impact_setup(m, 30.0, 1e-5)
    inst = [dict(xloc=m.xloc, conn=m.conn, E=E, nu=NU, rho=RHO, sigma_y0=100e6, H=0.689e9,
                 wall_normal=setup["wall_normal"], wall_offset=setup["wall_offset"],
                 wall_stiffness=setup["wall_stiffness"], vel=setup["vel"], dt=setup["dt"],
                 t_end=20.5 * setup["dt"])]
    out = []
    for second in (False, True):
        b = cilib.Batch(inst, **LARGE)
        c = cilib.Batch(inst, **SMALL) if second else None
        b.run()
        out.append(b.state(0))
        b.close()
        if c:
            c.run()
            c.close()
    for k in ("x", "v", "epbar", "contact"):
        assert np.array_equal(out[0][k], out[1][k]), k


def test_automatic_kernel_of_the_first_solver(cilib):
    """The automatic choice asks how many chunks fit an SM.  In a process of its own: the first
    solver, with chunks beyond the 48 KB that a kernel has by default, takes the kernel that
    any later one does (few chunks: the fused one)."""
    code = ("import sys; sys.path.insert(0, %r)\n"
            "from cppimpact_gb300 import api, meshgen as mg\n"
            "m = mg.cube(10, 2)\n"
            "k = [api.Solver(m.xloc, m.conn, E=1e9, nu=0.3, rho=1e3, chunk_nodes=n, chunk_elements=4096)"
            ".step_kernel() for n in (1400, 512, 1400)]\n"
            "print(k)\n" % ROOT)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ))
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.split("\n")[0] == "[3, 3, 3]"
