"""Performance cases of the impact framework: single solves, the drop-in driver, parameter
sweeps, the surrogate's training and answers, and the POD's products, each through the
package's public entry points on synthetic inputs made from a seed.

``listed()`` names the cases, ``draw(rng)`` gives one more of the same ranges,
``prepare(case, seed)`` builds what a program holds before the call, ``run(state)`` makes
one call, ``work(case)`` counts the bytes and operations the call needs, and
``exact(case, seed)`` evaluates the same formulation in 64 bits with plain torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cppimpact_gb300 import api
from cppimpact_gb300 import meshgen as mg
from cppimpact_gb300 import surrogate as sg
from cppimpact_gb300 import sweep as sw

E, NU, RHO = 68.9e9, 0.33, 2700.0
L2_BYTES = 129e6


def listed():
    return [
        # A host loop that exchanges the state with another code after every step, on the
        # smallest configured mesh (10^3 x 6 tet4): one step per call, latency only.
        dict(name="tet4_6k_step1", kind="run", mesh="cube", n=10, order=1, steps=1, mode="j2"),
        # The same mesh advanced between two reads of the state (an export interval).
        dict(name="tet4_6k_run200", kind="run", mesh="cube", n=10, order=1, steps=200, mode="j2"),
        # A driver written for the reference (initialize + solve + all fields back), its own
        # force law, a mesh of the size of its fuselage input (21,657 tet4).
        dict(name="dropin_tet4_20k", kind="dropin", n=15, order=1, steps=300),
        # The quadratic cube of the configurations: 34,992 tet10, yielding impact.
        dict(name="tet10_35k_run100", kind="run", mesh="cube", n=18, order=2, steps=100, mode="j2"),
        # A shell segment (720 x 20 cells, 86,400 tet10) with an odd number of steps.
        dict(name="tet10_86k_run25", kind="run", mesh="shell", n=720, axial=20, order=2, steps=25,
             mode="j2"),
        # The headline mesh: the 604,800-element tet10 shell, an export interval of 50 steps.
        dict(name="shell_605k_run50", kind="run", mesh="shell", n=720, axial=140, order=2, steps=50,
             mode="j2"),
        # A parameter sweep of uneven cubes of both element types (default tile shape, a
        # fifth of its 2 ms), end states read.
        dict(name="sweep_mixed24", kind="sweep", count=24, n_lo=6, n_hi=16, t_end=4e-4),
        # Training data of the surrogate: many 12^3 x 6 tet4 cubes with displacement snapshots,
        # in the tile shape that the autotuner reports for such a batch.
        dict(name="sweep_snaps64", kind="snaps", count=64, n=12, order=1, every=50, snaps=8,
             tuned=True),
        # Training one ensemble member of the surrogate (4 -> 256 -> 256 -> 64 x 80).
        dict(name="mlp_train_5120", kind="train", hidden=256, n_out=5120, rows=4096, batch=256,
             epochs=1),
        # 512 queries answered by a trained member: prediction and POD reconstruction.
        dict(name="surrogate_answer512", kind="answer", queries=512, hidden=256, snaps=80, rank=64,
             dofs=6591),
        # The POD range finder's sketch S Omega of 1,024 runs (rows of 6,591: not 16-byte
        # aligned) and its long projection S^T Q (aligned operands, K = rows).
        dict(name="pod_sketch_1024", kind="gemm", M=81920, N=96, K=6591, ta=0, tb=1),
        dict(name="pod_project_1024", kind="gemm", M=6591, N=96, K=81920, ta=0, tb=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "dropin", "sweep", "snaps", "train", "answer", "gemm",
                       "gemm"])
    if kind == "run":
        order = rng.choice([1, 2])
        steps = _log(rng, 1, 200)
        mode = rng.choice(["j2", "j2", "refcompat"])
        if rng.random() < 0.4:
            axial = _log(rng, 2, 100)
            return dict(kind=kind, mesh="shell", n=rng.randint(97, 720), axial=axial, order=order,
                        steps=min(steps, 50), mode=mode)
        return dict(kind=kind, mesh="cube", n=_log(rng, 3, 40 if order == 1 else 32), order=order,
                    steps=min(steps, 100), mode=mode)
    if kind == "dropin":
        return dict(kind=kind, n=_log(rng, 4, 20), order=1, steps=_log(rng, 20, 400))
    if kind == "sweep":
        lo = rng.randint(3, 8)
        return dict(kind=kind, count=_log(rng, 2, 24), n_lo=lo, n_hi=rng.randint(lo, 14),
                    t_end=rng.choice([1e-4, 2e-4]))
    if kind == "snaps":
        return dict(kind=kind, count=_log(rng, 4, 64), n=rng.randint(4, 12), order=1,
                    every=2 * rng.randint(5, 25), snaps=rng.randint(2, 8), tuned=rng.random() < 0.5)
    if kind == "train":
        return dict(kind=kind, hidden=rng.choice([64, 128, 256]), n_out=_log(rng, 1, 5120),
                    rows=_log(rng, 300, 4096), batch=rng.choice([128, 200, 256]), epochs=1)
    if kind == "answer":
        return dict(kind=kind, queries=_log(rng, 1, 512), hidden=256, snaps=rng.choice([40, 80]),
                    rank=rng.choice([32, 64]), dofs=3 * (rng.randint(6, 12) + 1) ** 3)
    # products of the POD and of the networks: tall, flat and odd, in the transpose forms
    # the package uses (A B^T, A B, A^T B)
    ta, tb = rng.choice([(0, 1), (0, 1), (0, 0), (1, 0)])
    return dict(kind="gemm", M=_log(rng, 64, 8192), N=_log(rng, 16, 512), K=_log(rng, 64, 16384),
                ta=ta, tb=tb)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _solve_inputs(case, seed):
    """Mesh (the same for every seed, as in a study of one part), impact set-up, material and
    initial nodal state of a single solve: a rigid impact velocity plus a smooth oscillation,
    so that the first steps already strain the body."""
    rng = np.random.default_rng(seed)
    if case["mesh"] == "shell":
        m = mg.shell(n_theta=case["n"], n_axial=case["axial"], L=4.0 * case["axial"] / 140.0,
                     order=case["order"])
        speed, gap, wave = rng.uniform(5.0, 20.0), 0.0, 0.5
    else:
        m = mg.cube(case["n"], case["order"])
        speed, gap, wave = rng.uniform(10.0, 30.0), 1e-4, 0.25
    setup = mg.impact_setup(m, speed, gap)
    k = 2.0 * np.pi / wave * rng.uniform(0.5, 1.5, size=(3, 3))
    ph = rng.uniform(0.0, 2.0 * np.pi, size=3)
    amp = 0.2 * speed
    v = np.asarray(setup["vel"])[None, :] + amp * np.sin(m.xloc @ k.T + ph)
    sy, H = rng.uniform(200e6, 350e6), rng.uniform(0.005, 0.02) * E
    return m, setup, np.ascontiguousarray(v), sy, H


def _dropin_inputs(case, seed):
    rng = np.random.default_rng(seed)
    m = mg.cube(case["n"], case["order"])
    setup = mg.impact_setup(m, rng.uniform(10.0, 30.0), 1e-4)
    return m, setup


def _sweep_inputs(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "sweep":
        # the sweep's parts are the same for every seed; speed, tilt and material are drawn
        out = sw.make_instances(case["count"], t_end=case["t_end"],
                                n_range=(case["n_lo"], case["n_hi"]))
        for d in out:
            c, s = math.cos(th := math.radians(rng.uniform(0.0, 15.0))), math.sin(th)
            d["wall_normal"] = (0.0, s, c)
            d["wall_offset"] = float((d["xloc"] @ np.array([0.0, s, c])).min() - 1e-3)
            d["vel"] = (0.0, 0.0, -float(rng.uniform(2.0, 20.0)))
            d["sigma_y0"], d["H"] = float(rng.uniform(200e6, 350e6)), float(rng.uniform(0.005, 0.02)) * E
        return out
    p = sg.sample_params(case["count"], rng)
    mesh = mg.cube(case["n"], case["order"])
    steps = case["every"] * case["snaps"]
    k, dt = mg.wall_stiffness(mesh, E), mg.cfl_dt(mesh, E, NU, RHO)
    out = []
    for v, sy, h, tilt in p:
        st = sw.tilted_setup(mesh, v, tilt, gap=1e-4, stiffness=k, dt=dt)
        st["t_end"] = (steps - 0.5) * dt
        out.append(dict(xloc=mesh.xloc, conn=mesh.conn, E=E, nu=NU, rho=RHO, sigma_y0=sy,
                        H=h * E, **st))
    return out


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _net_inputs(case, seed):
    g = _gen(seed)
    n_out = case["n_out"] if case["kind"] == "train" else case["snaps"] * case["rank"]
    rows = case["rows"] if case["kind"] == "train" else case["queries"]
    X = 2.0 * torch.rand((rows, 4), generator=g, device="cuda") - 1.0
    # smooth targets of the parameters, as the normalised modal trajectories are
    W = torch.randn((4, n_out), generator=g, device="cuda")
    T = 0.5 * torch.sin(2.0 * X @ W)
    return X.contiguous(), T.contiguous(), n_out


def _basis(case, seed):
    Q, _ = torch.linalg.qr(torch.randn((case["dofs"], case["rank"]), generator=_gen(seed + 1),
                                       device="cuda"))
    return Q.to(torch.bfloat16).contiguous()


def _gemm_inputs(case, seed):
    g = _gen(seed)
    M, N, K = case["M"], case["N"], case["K"]
    A = torch.randn((K, M) if case["ta"] else (M, K), generator=g, device="cuda",
                    dtype=torch.bfloat16)
    B = torch.randn((N, K) if case["tb"] else (K, N), generator=g, device="cuda",
                    dtype=torch.bfloat16)
    return A, B


def _snaps_batch(case, inst):
    shape = dict(chunk_elements=4096, chunk_nodes=512, block_threads=128) if case["tuned"] else {}
    return api.Batch(inst, **shape)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "run":
        m, setup, v, sy, H = _solve_inputs(case, seed)
        ref = case["mode"] == "refcompat"
        s = api.Solver(m.xloc, m.conn, E=E, nu=NU, rho=RHO, sigma_y0=sy, H=H,
                       mode=api.MODE_REFCOMPAT if ref else api.MODE_J2, lumping=api.LUMP_HRZ,
                       wall_normal=setup["wall_normal"], wall_offset=setup["wall_offset"],
                       wall_stiffness=setup["wall_stiffness"])
        s.initialize(setup["vel"])
        s.set_state(m.xloc, v)
        s.start(setup["dt"])
        # pinned host buffers the caller reads the state into
        xo = torch.empty((m.num_nodes, 3), dtype=torch.float64, pin_memory=True)
        vo = torch.empty((m.num_nodes, 3), dtype=torch.float64, pin_memory=True)
        return dict(kind=kind, s=s, steps=case["steps"], keep=(xo, vo), x=xo.numpy(), v=vo.numpy())
    if kind == "dropin":
        m, setup = _dropin_inputs(case, seed)
        mesh = api.Mesh(m.npe)
        mesh.num_nodes, mesh.num_elements = m.num_nodes, m.num_elements
        mesh.xloc, mesh.element_nodes, mesh.slave_nodes = m.xloc.reshape(-1), m.conn, m.slave
        mat = api.BaseMaterial("LinearElastic", E, RHO, NU)
        wall = api.Wall("wall", setup["wall_offset"], setup["wall_stiffness"], m.slave,
                        len(m.slave), 1)
        d = api.Dynamics(mesh, mat, wall)
        return dict(kind=kind, d=d, vel=setup["vel"], dt=setup["dt"],
                    t_end=(case["steps"] - 0.5) * setup["dt"])
    if kind == "sweep":
        inst = _sweep_inputs(case, seed)
        return dict(kind=kind, b=api.Batch(inst), n=len(inst))
    if kind == "snaps":
        inst = _sweep_inputs(case, seed)
        b = _snaps_batch(case, inst)
        buf = torch.zeros((case["snaps"], len(inst) * inst[0]["xloc"].shape[0], 3),
                          dtype=torch.float32, device="cuda")
        return dict(kind=kind, b=b, every=case["every"], snaps=case["snaps"], buf=buf)
    if kind == "train":
        X, T, n_out = _net_inputs(case, seed)
        net = sg.MLP(4, case["hidden"], n_out, seed + 1)
        return dict(kind=kind, net=net, X=X, T=T, epochs=case["epochs"], batch=case["batch"],
                    seed=seed)
    if kind == "answer":
        X, _, n_out = _net_inputs(case, seed)
        net = sg.MLP(4, case["hidden"], n_out, seed + 1)
        return dict(kind=kind, net=net, X=X, Phib=_basis(case, seed), rank=case["rank"])
    A, B = _gemm_inputs(case, seed)
    return dict(kind=kind, A=A, B=B, ta=bool(case["ta"]), tb=bool(case["tb"]))


def run(state):
    kind = state["kind"]
    if kind == "run":
        state["s"].step(state["steps"])
        state["s"].get_xv(state["x"], state["v"])
        return dict(x=state["x"], v=state["v"])
    if kind == "dropin":
        state["d"].initialize((0.0, 0.0, 0.0), state["vel"])
        return state["d"].solve(state["dt"], state["t_end"])
    if kind == "sweep":
        state["b"].run()
        st = [state["b"].state(i) for i in range(state["n"])]
        return {k: np.concatenate([s[k].reshape(-1) for s in st])
                for k in ("x", "v", "epbar", "contact")}
    if kind == "snaps":
        state["b"].run_snapshots(state["every"], state["buf"].data_ptr(), state["snaps"])
        return state["buf"]
    if kind == "train":
        loss = state["net"].train(state["X"], state["T"], state["epochs"], state["batch"], 2e-3,
                                  state["seed"])
        return dict(loss=loss, params=state["net"].params())
    if kind == "answer":
        Y = state["net"].predict(state["X"])
        A = Y.view(-1, state["rank"]).to(torch.bfloat16)
        return dict(Y=Y, U=sg.gemm(A, state["Phib"], transB=True))
    return sg.gemm(state["A"], state["B"], transA=state["ta"], transB=state["tb"])


# ---------------------------------------------------------------------------
# Work
# ---------------------------------------------------------------------------

def _mesh_size(kind, n, order, axial=None):
    """(elements, nodes) of the generated meshes."""
    if kind == "shell":
        cells = n * axial
        edges_v = 2 * n * (axial + 1)
        # tet10: (2 n) x (2 axial + 1) x 3 lattice of the periodic strip
        return 6 * cells, (2 * n) * (2 * axial + 1) * 3 if order == 2 else edges_v
    side = 2 * n + 1 if order == 2 else n + 1
    return 6 * n ** 3, side ** 3


def _step_work(El, N, order, steps):
    """Element state (connectivity, stress and plastic strain in and out) and node state
    of a step, moved once per step where the mesh does not fit the L2 and once per call
    where it does; operations per step at about 600 (tet10: four points) per point."""
    npe, nq = (4, 1) if order == 1 else (10, 4)
    b = El * (4 * npe + 56 * nq) + 112 * N
    return b * (steps if b > L2_BYTES else 1), (El * nq * 600.0 + N * 30.0) * steps


def work(case):
    kind = case["kind"]
    if kind == "run":
        El, N = _mesh_size(case["mesh"], case["n"], case["order"], case.get("axial"))
        b, f = _step_work(El, N, case["order"], case["steps"])
        return dict(bytes=b + 48 * N, flops=f)
    if kind == "dropin":
        El, N = _mesh_size("cube", case["n"], case["order"])
        b, f = _step_work(El, N, case["order"], case["steps"])
        return dict(bytes=b + 57 * N + 28 * El, flops=f)
    if kind in ("sweep", "snaps"):
        tot_b, tot_f = 0.0, 0.0
        if kind == "snaps":
            El, N = _mesh_size("cube", case["n"], case["order"])
            El, N = El * case["count"], N * case["count"]
            b, f = _step_work(El, N, case["order"], case["every"] * case["snaps"])
            return dict(bytes=b + 12 * N * case["snaps"], flops=f)
        for order in (1, 2):
            ns = range(case["n_lo"], case["n_hi"] + 1)
            for n in ns:   # expected mix: sizes and element types uniform
                El, N = _mesh_size("cube", n, order)
                h = 0.25 / n * 0.45 * (0.5 if order == 2 else 1.0)
                steps = case["t_end"] / (0.5 * h / mg.dilatational_speed(E, NU, RHO))
                b, f = _step_work(El, N, order, steps)
                tot_b += (b + 49 * N) / (2 * len(ns))
                tot_f += f / (2 * len(ns))
        return dict(bytes=tot_b * case["count"], flops=tot_f * case["count"])
    if kind in ("train", "answer"):
        H = case["hidden"]
        n_out = case["n_out"] if kind == "train" else case["snaps"] * case["rank"]
        P = 4 * H + H + H * H + H + H * n_out + n_out
        if kind == "train":
            batches = max(1, case["rows"] // case["batch"]) * case["epochs"]
            rows = min(case["rows"], case["batch"])
            return dict(bytes=batches * rows * (16.0 + 4 * n_out) + 24.0 * P,
                        flops=batches * 6.0 * rows * P)
        rows = case["queries"]
        U = rows * case["snaps"] * case["dofs"]
        return dict(bytes=4.0 * P + rows * n_out * 4.0 + 2.0 * case["dofs"] * case["rank"] + 4.0 * U,
                    flops=2.0 * rows * P + 2.0 * U * case["rank"])
    M, N, K = case["M"], case["N"], case["K"]
    return dict(bytes=2.0 * (M * K + N * K) + 4.0 * M * N, flops=2.0 * M * N * K)


# ---------------------------------------------------------------------------
# The same results in 64 bits
# ---------------------------------------------------------------------------

def _rule(npe):
    """Shape-function gradients [nq, npe, 3], values [nq, npe] and weight."""
    if npe == 4:
        G = np.array([[-1.0, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]])
        return G[None], np.full((1, 4), 0.25), 1.0 / 6.0
    dL = np.array([[1.0, 0, 0], [0, 1.0, 0], [-1.0, -1.0, -1.0], [0, 0, 1.0]])
    a, b = (5 + 3 * np.sqrt(5)) / 20, (5 - np.sqrt(5)) / 20
    edges = [(0, 1), (1, 2), (2, 0), (0, 3), (1, 3), (2, 3)]
    G, S = [], []
    for q in range(4):
        L = [a if q == 1 else b, a if q == 2 else b, a if q == 0 else b, a if q == 3 else b]
        G.append([(4 * L[c] - 1) * dL[c] for c in range(4)] +
                 [4 * (L[i] * dL[j] + L[j] * dL[i]) for i, j in edges])
        S.append([L[c] * (2 * L[c] - 1) for c in range(4)] + [4 * L[i] * L[j] for i, j in edges])
    return np.array(G), np.array(S), 1.0 / 24.0


def _inv3(J):
    c = torch.stack([torch.linalg.cross(J[..., 1, :], J[..., 2, :]),
                     torch.linalg.cross(J[..., 2, :], J[..., 0, :]),
                     torch.linalg.cross(J[..., 0, :], J[..., 1, :])], dim=-1)
    det = (J[..., 0, :] * c[..., :, 0]).sum(-1)
    return c / det[..., None, None], det


class _Solve64:
    """The explicit impact run in FP64 for instances of one element type held as one mesh;
    parameters are per instance, expanded to elements and nodes."""

    def __init__(self, meshes, pars, mode, lumping):
        dev = "cuda"
        self.npe = meshes[0][1].shape[1]
        G, S, self.W = _rule(self.npe)
        self.G = torch.tensor(G, device=dev)
        off, X, conn, ie, inn = 0, [], [], [], []
        for i, (x, c) in enumerate(meshes):
            X.append(x)
            conn.append(c.astype(np.int64) + off)
            off += x.shape[0]
            ie.append(np.full(c.shape[0], i))
            inn.append(np.full(x.shape[0], i))
        t = lambda a: torch.tensor(np.concatenate(a), device=dev)
        self.X, self.conn, self.ie, self.inn = t(X), t(conn), t(ie), t(inn)
        g = lambda k: torch.tensor(np.array([p[k] for p in pars], dtype=np.float64), device=dev)
        self.dt, self.wk, self.woff, self.wn = g("dt"), g("k"), g("off"), g("n")
        self.sy, self.H = g("sy"), g("H")
        self.nsteps = torch.tensor([p["steps"] for p in pars], device=dev)
        self.mode = mode
        self.lam, self.mu = E * NU / ((1 + NU) * (1 - 2 * NU)), E / (2 * (1 + NU))
        self.grav = torch.tensor([0.0, 0.0, -9.81], device=dev, dtype=torch.float64)
        self.v = t([np.broadcast_to(p["v"], m[0].shape) for p, m in zip(pars, meshes)]).clone()
        self.u = torch.zeros_like(self.X)
        nE, nq = self.conn.shape[0], self.G.shape[0]
        self.sig = torch.zeros((nE, nq, 3, 3), device=dev, dtype=torch.float64)
        self.ep = torch.zeros((nE, nq), device=dev, dtype=torch.float64)
        _, _, wd = self._geom()
        if lumping == "hrz" and self.npe == 10:
            V = RHO * wd.sum(1)
            me = torch.cat([V[:, None].expand(-1, 4) / 36.0, V[:, None].expand(-1, 6) * 4.0 / 27.0], 1)
        else:
            me = RHO * wd @ torch.tensor(S, device=dev)
        self.mass = torch.zeros(off, device=dev, dtype=torch.float64)
        self.mass.index_add_(0, self.conn.reshape(-1), me.reshape(-1))
        a = self._wall(self.grav.expand_as(self.u).clone(), self.u)
        self.v += 0.5 * self.dt[self.inn][:, None] * a

    def _geom(self):
        x = (self.X + self.u)[self.conn]
        J = torch.einsum("eia,qij->eqaj", x - x[:, :1], self.G)
        Ji, det = _inv3(J)
        return x, Ji, self.W * det

    def _wall(self, a, u):
        n = self.wn[self.inn]
        d = ((self.X + u) * n).sum(1) - self.woff[self.inn]
        c = torch.where(d < 0, -d * self.wk[self.inn] / self.mass, torch.zeros_like(d))
        return a + c[:, None] * n

    def step(self, k):
        act_e, act_n = (k < self.nsteps)[self.ie], (k < self.nsteps)[self.inn]
        dtn = self.dt[self.inn][:, None]
        _, Ji, wd = self._geom()
        L = torch.einsum("eia,qij->eqaj", (dtn * self.v)[self.conn], self.G) @ Ji
        de = 0.5 * (L + L.transpose(-1, -2))
        tr = de.diagonal(dim1=-2, dim2=-1).sum(-1)
        eye = torch.eye(3, device=L.device, dtype=torch.float64)
        ds = self.lam * tr[..., None, None] * eye + 2 * self.mu * de
        if self.mode == "j2":
            s = self.sig + ds
            pm = s.diagonal(dim1=-2, dim2=-1).sum(-1)[..., None, None] / 3 * eye
            d = s - pm
            nrm = d.square().sum((-1, -2)).sqrt()
            sy, H = self.sy[self.ie][:, None], self.H[self.ie][:, None]
            r = math.sqrt(2.0 / 3.0)
            f = nrm - r * (sy + H * self.ep)
            dg = torch.where(f > 0, f / (2 * self.mu + 2.0 / 3.0 * H), torch.zeros_like(f))
            s = d * (1 - 2 * self.mu * dg / nrm.clamp_min(1e-300))[..., None, None] + pm
            m = act_e[:, None]
            self.sig = torch.where(m[..., None, None], s, self.sig)
            self.ep = torch.where(m, self.ep + r * dg, self.ep)
        else:
            s = ds
        P = wd[..., None, None] * (s @ Ji.transpose(-1, -2))
        fe = torch.einsum("eqaj,qij->eia", P, self.G)
        f = torch.zeros_like(self.u)
        f.index_add_(0, self.conn.reshape(-1), fe.reshape(-1, 3))
        un = self.u + dtn * self.v
        a = self._wall(self.grav - f / self.mass[:, None], un)
        m = act_n[:, None]
        self.v = torch.where(m, self.v + dtn * a, self.v)
        self.u = torch.where(m, un, self.u)


def _voigt(s):
    return torch.stack([s[..., 0, 0], s[..., 1, 1], s[..., 2, 2], s[..., 0, 1], s[..., 1, 2],
                        s[..., 0, 2]], dim=-1)


def _exact_sweep(case, seed):
    inst = _sweep_inputs(case, seed)
    done = {}
    for npe in (4, 10):
        ids = [i for i, d in enumerate(inst) if d["conn"].shape[1] == npe]
        if not ids:
            continue
        pars = []
        for i in ids:
            d = inst[i]
            steps, t = 0, 0.0
            while t <= d["t_end"]:
                steps, t = steps + 1, t + d["dt"]
            pars.append(dict(dt=d["dt"], k=d["wall_stiffness"], off=d["wall_offset"],
                             n=d["wall_normal"], sy=d["sigma_y0"], H=d["H"], steps=steps,
                             v=np.asarray(d["vel"])))
        S = _Solve64([(inst[i]["xloc"], inst[i]["conn"]) for i in ids], pars, "j2", "hrz")
        snaps = []
        for k in range(int(S.nsteps.max())):
            S.step(k)
            if case["kind"] == "snaps" and (k + 1) % case["every"] == 0:
                snaps.append(S.u.clone())
        if case["kind"] == "snaps":
            return S, torch.stack(snaps)
        for j, i in enumerate(ids):
            mn, me = S.inn == j, S.ie == j
            done[i] = ((S.X + S.u)[mn], S.v[mn], S.ep[me])
    cat = lambda k: torch.cat([done[i][k].reshape(-1) for i in range(len(inst))])
    return dict(x=cat(0), v=cat(1), epbar=cat(2), contact=None)


def exact(case, seed):
    kind = case["kind"]
    if kind == "run":
        m, setup, v, sy, H = _solve_inputs(case, seed)
        par = dict(dt=setup["dt"], k=setup["wall_stiffness"], off=setup["wall_offset"],
                   n=setup["wall_normal"], sy=sy, H=H, steps=case["steps"], v=v)
        S = _Solve64([(m.xloc, m.conn)], [par], case["mode"], "hrz")
        for k in range(case["steps"]):
            S.step(k)
        return dict(x=S.X + S.u, v=S.v)
    if kind == "dropin":
        m, setup = _dropin_inputs(case, seed)
        par = dict(dt=setup["dt"], k=setup["wall_stiffness"], off=setup["wall_offset"],
                   n=setup["wall_normal"], sy=0.0, H=0.0, steps=case["steps"],
                   v=np.asarray(setup["vel"]))
        S = _Solve64([(m.xloc, m.conn)], [par], "refcompat", "rowsum")
        for k in range(case["steps"]):
            S.step(k)
        return dict(x=S.X + S.u, v=S.v, mass=S.mass, sigma=None, epbar=None, contact=None)
    if kind == "sweep":
        return _exact_sweep(case, seed)
    if kind == "snaps":
        # the run's snapshot buffer is in the library's node order
        S, u = _exact_sweep(case, seed)
        inst = _sweep_inputs(case, seed)
        b = _snaps_batch(case, inst)
        N = inst[0]["xloc"].shape[0]
        order = np.concatenate([b.node_order(i)[0] + i * N for i in range(len(inst))])
        b.close()
        return u[:, torch.tensor(order, device="cuda", dtype=torch.int64)]
    if kind == "train":
        return None   # the mini-batch order is the library's own generator's
    if kind == "answer":
        X, _, n_out = _net_inputs(case, seed)
        net = sg.MLP(4, case["hidden"], n_out, seed + 1)
        p = torch.tensor(net.params(), device="cuda", dtype=torch.float64)
        H = case["hidden"]
        parts = torch.split(p, [4 * H, H, H * H, H, H * n_out, n_out])
        h = torch.tanh(X.double() @ parts[0].view(4, H) + parts[1])
        h = torch.tanh(h @ parts[2].view(H, H) + parts[3])
        Y = h @ parts[4].view(H, n_out) + parts[5]
        return dict(Y=Y, U=Y.view(-1, case["rank"]) @ _basis(case, seed).double().t())
    A, B = _gemm_inputs(case, seed)
    A = A.t() if case["ta"] else A
    B = B.t() if case["tb"] else B
    out = torch.zeros((case["M"], case["N"]), device="cuda", dtype=torch.float64)
    for k in range(0, case["K"], 8192):
        out += A[:, k:k + 8192].double() @ B[k:k + 8192].double()
    return out
