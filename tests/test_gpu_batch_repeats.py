"""Batches of tet10 meshes with an element that names a node twice, in the forms the batch may
take: chunks held on the SMs, whose element forces have an entry per corner, and a launch per
step, whose four lanes must not share an accumulator."""
import numpy as np
import pytest

from cppimpact_gb300 import meshgen as mg

pytestmark = pytest.mark.gpu

MAT = dict(E=68.9e9, nu=0.33, rho=2700.0, sigma_y0=100e6, H=0.689e9)


def repeated(m, every):
    """Every `every`-th element's first edge node is its first corner (its Jacobian stays
    positive at the Gauss points); nodes that no element names any more go."""
    conn = m.conn.copy()
    conn[::every, 4] = conn[::every, 0]
    used, inverse = np.unique(conn, return_inverse=True)
    return m.xloc[used].copy(), inverse.reshape(conn.shape).astype(np.int32)


def instance(x, conn, m, speed, steps, dt_scale):
    setup = mg.impact_setup(m, speed, 1e-5)
    dt = dt_scale * setup["dt"]
    return dict(xloc=x, conn=conn, **MAT, wall_normal=setup["wall_normal"],
                wall_offset=setup["wall_offset"], wall_stiffness=setup["wall_stiffness"],
                vel=setup["vel"], dt=dt, t_end=(steps - 0.5) * dt)


@pytest.mark.parametrize("mesh,shape", [("cube", {}), ("cube", dict(chunk_elements=700)),
                                        ("apart", dict(chunk_elements=60))])
def test_repeated_node_in_batch(cilib, mesh, shape):
    """Against single solves of the same plan.  "apart": tetrahedra that share no node, 600
    nodes in a chunk of 60, more chunks than the GPU holds at once; by itself an element with
    a repeated node has eigenfrequencies up to 1.94 / dt, beside the wall's 0.98 / dt beyond
    what the step integrates, so there the step is a quarter.  The kernels may fuse different
    products, 1e-6 of a force per step: velocities agree to 1e-5 of the largest.  A lost
    update is the force of an element on a node, 1e-2 and more of a velocity that the wall
    turns round."""
    steps, dt_scale = (120, 0.25) if mesh == "apart" else (30, 1.0)
    m = mg.cube(15 if mesh == "apart" else 9, 2)
    if mesh == "apart":
        m.xloc = m.xloc[m.conn.reshape(-1)].copy()
        m.conn = np.arange(m.conn.size, dtype=np.int32).reshape(m.conn.shape)
    x, conn = repeated(m, 50)
    inst = [instance(x, conn, m, v, steps, dt_scale) for v in (20.0, 30.0)]
    b = cilib.Batch(inst, **shape)
    b.run()
    for i, d in enumerate(inst):
        s = cilib.Solver(x, conn, **MAT, wall_normal=d["wall_normal"], wall_offset=d["wall_offset"],
                         wall_stiffness=d["wall_stiffness"], elem_lanes=1, step_kernel=1, **shape)
        s.initialize(d["vel"])
        s.start(d["dt"])
        s.step(steps)
        a, g = s.state(), b.state(i)
        assert (a["contact"] & 2).any() and np.array_equal(a["contact"], g["contact"])
        for k in ("x", "v"):
            scale = np.abs(a[k] - (d["xloc"] if k == "x" else 0.0)).max()
            assert np.abs(a[k] - g[k]).max() <= 1e-5 * scale, k
        s.close()
    b.close()
