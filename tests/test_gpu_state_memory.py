"""A state read into page-locked memory that is made of several registrations."""
import ctypes as C
import mmap

import numpy as np
import pytest

from cppimpact_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu


def test_adjacent_registrations(cilib):
    """8,000 nodes, 192,000 bytes, across a boundary between two registrations: every byte is
    page-locked, no one registration holds the array."""
    torch = pytest.importorskip("torch")
    m = mg.cube(19, 1)
    setup = mg.impact_setup(m, 20.0, 0.0)
    s = cilib.Solver(m.xloc, m.conn, E=68.9e9, nu=0.33, rho=2700.0, sigma_y0=276e6, H=0.689e9,
                     wall_normal=setup["wall_normal"],
                     wall_offset=setup["wall_offset"], wall_stiffness=setup["wall_stiffness"])
    s.initialize(setup["vel"])
    s.start(setup["dt"])
    s.step(3)
    x, v = np.empty((m.num_nodes, 3)), np.empty((m.num_nodes, 3))
    s.get_xv(x, v)
    half = 1 << 20
    mem = mmap.mmap(-1, 3 * half)
    base = C.addressof(C.c_char.from_buffer(mem))
    first = -(-base // half) * half   # on a page boundary, whatever a page is
    rt = torch.cuda.cudart()
    for at in (first, first + half // 2):
        assert int(rt.cudaHostRegister(at, half // 2, 0)) == 0
    try:
        n = 3 * m.num_nodes
        pinned = np.ctypeslib.as_array((C.c_double * (half // 8)).from_address(first))
        pinned[:] = 7.0
        lo = half // 16 - n // 2
        px = pinned[lo:lo + n]
        s.get_xv(px, v)
        assert np.array_equal(px, x.ravel())
        assert (pinned[:lo] == 7.0).all() and (pinned[lo + n:] == 7.0).all()
    finally:
        for at in (first, first + half // 2):
            rt.cudaHostUnregister(at)
    s.close()
