"""The resident form of the fused step: the bits of the launch-per-step form on the same
plan, at the sizes where its chunks change form, and the batch's snapshots."""
import numpy as np
import pytest

from cppimpact_gb300 import meshgen as mg
from cppimpact_gb300 import sweep

pytestmark = pytest.mark.gpu

E, NU, RHO = 68.9e9, 0.33, 2700.0


@pytest.mark.parametrize("order,n,mode", [(1, 15, "j2"), (1, 19, "refcompat"), (1, 30, "j2"),
                                          (2, 13, "j2"), (2, 18, "refcompat"), (2, 18, "j2")])
def test_resident_equals_launch_per_step(cilib, order, n, mode):
    """Chunks of 34, 68 and 267 tet4 and 22 and 58 tet10 elements, through a yielding
    contact: 64-thread CTAs leave the resident form where a thread of the 64 would have
    more than one element or point (the same plan, one launch per step), and the state does
    not depend on the CTA size."""
    m = mg.cube(n, order)
    setup = mg.impact_setup(m, 30.0, 1e-5)
    out = []
    for bs in (128, 64):
        s = cilib.Solver(m.xloc, m.conn, E=E, nu=NU, rho=RHO, sigma_y0=100e6, H=0.689e9,
                         mode=cilib.MODE_J2 if mode == "j2" else cilib.MODE_REFCOMPAT,
                         lumping=cilib.LUMP_HRZ, wall_normal=setup["wall_normal"],
                         wall_offset=setup["wall_offset"],
                         wall_stiffness=setup["wall_stiffness"], block_threads=bs, step_kernel=3)
        s.initialize(setup["vel"])
        s.start(setup["dt"])
        for k in (1, 2, 41, 60):
            s.step(k)
        out.append((s.state(), s.nodal_fields()["acc"]))
        s.close()
    (a, acc_a), (b, acc_b) = out
    assert (a["contact"] & 2).any()
    for k in ("x", "v", "sigma", "epbar", "contact"):
        assert np.array_equal(a[k], b[k]), k
    assert np.array_equal(acc_a, acc_b)


@pytest.mark.parametrize("order,shape", [(1, {}), (2, {}), (2, dict(chunk_elements=4096,
                                                                   chunk_nodes=400))])
def test_batch_snapshots_and_peaks(cilib, order, shape):
    """Instances of uneven size and length: snapshot s is the state after 10 (s + 1) steps,
    or the last state of an instance that has ended; the peaks are the snapshots' largest
    displacement and the final plastic strain.  Displacements recovered from the solver's
    FP64 positions carry 1e-16 of the 0.25 m coordinates against 1e-7 m, so FP32 values
    agree to 1e-6."""
    torch = pytest.importorskip("torch")
    inst = [d for d in sweep.make_instances(12, t_end=1e-4, n_range=(2, 5), seed=3)
            if d["order"] == order][:4]
    for j, d in enumerate(inst):
        d["wall_offset"] += 9.9e-4
        d["t_end"] = (10 * j + 13 - 0.5) * d["dt"]
    b = cilib.Batch(inst, **shape)
    n_all = sum(d["xloc"].shape[0] for d in inst)
    snaps = 6
    buf = torch.zeros((snaps, n_all, 3), device="cuda")
    b.run_snapshots(10, buf.data_ptr(), snaps)
    got = buf.cpu().numpy()
    pd, pe, _ = b.run_peaks(10, snaps)
    longest = 10 * (len(inst) - 1) + 13
    written = min(snaps, longest // 10 + 1)
    for i, d in enumerate(inst):
        perm, off = b.node_order(i)
        s = cilib.Solver(d["xloc"], d["conn"], E=d["E"], nu=d["nu"], rho=d["rho"],
                         sigma_y0=d["sigma_y0"], H=d["H"], wall_normal=d["wall_normal"],
                         wall_offset=d["wall_offset"], wall_stiffness=d["wall_stiffness"], **shape)
        s.initialize(d["vel"])
        s.start(d["dt"])
        left = 10 * i + 13
        peak = 0.0
        for k in range(written):
            s.step(min(10, left))
            left -= min(10, left)
            u = (s.state(("x",))["x"] - d["xloc"])[perm]
            g = got[k, off:off + len(perm)]
            assert np.linalg.norm(g - u) <= 1e-6 * np.linalg.norm(u), (i, k)
            peak = max(peak, float(np.linalg.norm(g.astype(np.float64), axis=1).max()))
        assert pd[i] == pytest.approx(peak, rel=1e-6)
        assert pe[i] == s.state(("epbar",))["epbar"].max()
        s.close()
    assert not got[written:].any()
    b.close()
