"""Timed workloads of the framework, through its public entry points.

A case is a dict of plain values. ``listed()`` names the ones that stand for the framework's work,
``draw(rng)`` gives another one of the same ranges; ``prepare`` builds what a program holds before
the call, ``run`` makes one pass, ``work`` states what a pass cannot do without, and ``exact`` gives
the outputs in 64 bits from plain torch and numpy.

Kinds of case:

* ``driver``   Driver::solve's own loop on a small mesh: the state in, then calc_timestep and step
               with the host in between, the solution out.
* ``advance``  a transient or relaxing run: a state uploaded, many steps without the host, the
               state read back through a snapshot.
* ``steady``   the sweep: several bump channels in one batched mesh, local time stepping in the
               mixed form that converges like FP64, and the surrogate's training targets out.
* ``train``    Adam steps of the surrogate network; ``predict`` its evaluation on a mesh's cells.
* ``wall``     the wall distance of every cell, the warm start's costliest input feature.
* ``mesh``     the face-based grid of a tetrahedral mesh, built on the GPU.
"""
from functools import lru_cache

import numpy as np
import torch

from netflux_b200 import meshgen as mg
from netflux_b200 import solver as S
from netflux_b200 import surrogate as sur

GAMMA = 1.4
N_PARAM_USED = 128 * 8 + 3 * 128 * 128 + 3 * 128 + 5 * 128 + 5  # weights and biases of the network


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _flow(kind, mesh, nx, ny, nz, steps, precision="fp64", lts=False, order="Second", scheme="TVD_RK3",
          limiter="Barth", name=None):
    c = {"kind": kind, "mesh": mesh, "nx": nx, "ny": ny, "nz": nz, "steps": steps, "precision": precision,
         "lts": lts, "order": order, "scheme": scheme, "limiter": limiter}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a first small run or a unit study: 6,000 tets, the host between the steps, launches count
        _flow("driver", "cube", 10, 10, 10, 10, name="driver_cube_6k"),
        # the unit cube with a density bump, 20^3 hexes: fits the L2, global time step
        _flow("advance", "cube", 20, 20, 20, 50, name="cube_48k"),
        # the shock tube, 400 x 8 x 8 hexes: global time step, limiter active at the shock
        _flow("advance", "sod", 400, 8, 8, 50, name="sod_154k"),
        # the large bump channel, 128 x 64 x 64 hexes (3,145,728 tets): local time stepping, HBM-resident
        _flow("advance", "bump", 128, 64, 64, 20, lts=True, name="bump_3m"),
        # the reference's other schemes on a ragged mesh: first order in space, explicit Euler in time
        _flow("advance", "cube", 31, 29, 33, 60, order="First", scheme="ExplicitEuler", name="first_order_178k"),
        # the fast transient form (FP32 copies) on the 96 x 48 x 48 channel, unlimited range of the solver
        _flow("advance", "bump", 96, 48, 48, 100, precision="mixed32", lts=True, name="bump_mixed32_1m"),
        # the sweep's batched solve, unlimited scheme: eight channels of 16 to 40 hexes in x
        {"kind": "steady", "cases": 8, "nx_lo": 16, "nx_hi": 40, "steps": 200, "check": 100, "ratchet": 0,
         "pick": 5, "name": "sweep_unlimited"},
        # the same with the Barth limiter and the ratchet on, fewer and larger channels
        {"kind": "steady", "cases": 4, "nx_lo": 32, "nx_hi": 56, "steps": 200, "check": 50, "ratchet": 50,
         "pick": 6, "name": "sweep_ratchet"},
        # surrogate training at the sweep's batch size
        {"kind": "train", "samples": 400000, "batch": 65536, "steps": 10, "name": "train_65536"},
        # warm-start prediction on a mesh's cells, a ragged count
        {"kind": "predict", "samples": 1000003, "name": "predict_1m"},
        # wall distance of the 96 x 48 x 48 channel
        {"kind": "wall", "nx": 96, "ny": 48, "nz": 48, "name": "wall_distance_1m"},
        # the grid of the 64 x 32 x 32 channel from nodes, tetrahedra and markers
        {"kind": "mesh", "nx": 64, "ny": 32, "nz": 32, "name": "mesh_build_393k"},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["driver", "advance", "advance", "advance", "advance", "advance", "steady", "steady",
                       "train", "predict", "wall", "mesh"])
    if kind == "driver":
        n = _log_int(rng, 6, 22)
        return _flow("driver", "cube", n, n + rng.randrange(3), n, rng.randrange(5, 16))
    if kind == "advance":
        form = rng.choice(["cube", "sod", "bump", "bump32", "first"])
        if form == "sod":
            ny = rng.randrange(4, 13)
            return _flow("advance", "sod", _log_int(rng, 100, 600), ny, ny + rng.randrange(3), rng.randrange(20, 61))
        if form == "cube":
            n = _log_int(rng, 9, 60)
            return _flow("advance", "cube", n, n + rng.randrange(4), n + 1, rng.randrange(20, 51),
                         limiter=rng.choice(["Barth", "Barth", "NONE"]))
        if form == "first":
            n = _log_int(rng, 9, 50)
            return _flow("advance", "cube", n + 1, n, n + rng.randrange(4), rng.randrange(20, 61), order="First",
                         scheme=rng.choice(["ExplicitEuler", "TVD_RK3"]))
        nx = _log_int(rng, 20, 112)
        return _flow("advance", "bump", nx, nx // 2 + rng.randrange(2), nx // 2, rng.randrange(16, 41), lts=True,
                     precision="mixed32" if form == "bump32" else "fp64", limiter=rng.choice(["Barth", "NONE"]))
    if kind == "steady":
        lo = rng.randrange(12, 33)
        return {"kind": "steady", "cases": rng.randrange(1, 6), "nx_lo": lo, "nx_hi": lo + rng.randrange(2, 16),
                "steps": rng.randrange(80, 151), "check": rng.choice([25, 40, 50]),
                "ratchet": rng.choice([0, 30]), "pick": rng.randrange(1000)}
    if kind == "train":
        return {"kind": "train", "samples": _log_int(rng, 20000, 600000), "batch": _log_int(rng, 1000, 65536),
                "steps": rng.randrange(4, 11)}
    if kind == "predict":
        return {"kind": "predict", "samples": _log_int(rng, 1000, 1500000)}
    nx = _log_int(rng, 16, 80)
    return {"kind": kind, "nx": nx, "ny": nx // 2 + rng.randrange(3), "nz": nx // 2}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@lru_cache(maxsize=16)
def _tets(mesh, nx, ny, nz, h=0.1):
    if mesh == "cube":
        return mg.box_tet_mesh(nx, ny, nz, jitter=0.1, seed=1234)
    if mesh == "sod":
        return mg.sod_mesh(nx, ny, nz)
    return mg.bump_mesh(nx, ny, nz, h=h)


@lru_cache(maxsize=16)
def _grid(mesh, nx, ny, nz, h=0.1):
    return S.Mesh.from_tet_mesh(_tets(mesh, nx, ny, nz, h))


def _freestream(c):
    if c["mesh"] == "cube":
        return (1.0, 0.5, 0.0, 0.0, 1.0 / GAMMA)
    return mg.SOD_LEFT if c["mesh"] == "sod" else mg.bump_freestream(0.5)


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _initial_state(c, seed):
    """Conserved variables [n_cells][5]: the free stream (the cube's density bump, the tube's two
    states) with smooth disturbances of a few percent, as a flow in development has them."""
    t = _tets(c["mesh"], c["nx"], c["ny"], c["nz"])
    x = torch.from_numpy(t.centroids()).to(_device())
    rng = np.random.default_rng(seed)
    fs = _freestream(c)
    V = torch.tensor(fs, dtype=torch.float64, device=x.device).repeat(x.shape[0], 1)
    if c["mesh"] == "cube":
        V[:, 0] += rng.uniform(0.05, 0.15) * torch.exp(-((x - 0.5) ** 2).sum(1) / (2 * 0.1 ** 2))
    if c["mesh"] == "sod":
        right = x[:, 0] > rng.uniform(0.4, 0.6)
        V[right] = torch.tensor(mg.SOD_RIGHT, dtype=torch.float64, device=x.device)
    sound = torch.sqrt(GAMMA * V[:, 4] / V[:, 0])
    for k in range(5):
        wave = torch.zeros(x.shape[0], dtype=torch.float64, device=x.device)
        for _ in range(3):
            w = torch.tensor(rng.uniform(-7.0, 7.0, 3), device=x.device)
            wave += rng.uniform(0.003, 0.01) * torch.sin(x @ w + rng.uniform(0, 6.28))
        V[:, k] += wave * (sound if 1 <= k <= 3 else V[:, k])
    return _conserved(V).cpu().numpy()


def _config(c):
    fs = _freestream(c)
    more = {}
    if c["mesh"] == "sod":  # each end keeps its own far field
        more = {"patch_farfield": {"left": mg.SOD_LEFT, "right": mg.SOD_RIGHT}, "farfield_density_fix": True}
    return S.Config(precision=c["precision"], CFL=0.8, local_time_stepping=c["lts"], density_fs=fs[0],
                    velocity_fs=list(fs[1:4]), pressure_fs=fs[4], spatial_order=c["order"],
                    time_scheme=c["scheme"], limiter=c["limiter"], **more)


def _channels(c, seed):
    """The sweep's channels: resolution and bump height belong to the case, the Mach number to the seed."""
    rng = np.random.default_rng(c["pick"])
    out = []
    for _ in range(c["cases"]):
        nx = int(rng.integers(c["nx_lo"], c["nx_hi"] + 1))
        out.append({"nx": nx + nx % 2, "h": round(float(rng.uniform(0.05, 0.11)), 4)})
    rng = np.random.default_rng(seed)
    for ch in out:
        ch["mach"] = float(rng.uniform(0.3, 0.55))
    return out


def _pinned(a):
    t = torch.from_numpy(np.ascontiguousarray(a))
    return t.pin_memory().numpy() if torch.cuda.is_available() else t.numpy()


def _network(seed):
    """FP32 parameters in the library's layout, uniform with the layers' fan-in."""
    rng = np.random.default_rng(seed)
    u = lambda shape, fan: rng.uniform(-1, 1, shape) / np.sqrt(fan)
    W0 = np.zeros((128, 16))
    W0[:, :8] = u((128, 8), 7)  # column 7: the bias
    W4 = np.zeros((16, 128))
    W4[:5] = u((5, 128), 128)
    b4 = np.zeros(16)
    b4[:5] = u(5, 128)
    return np.concatenate([W0.ravel(), u(3 * 128 * 128, 128), u(3 * 128, 128), W4.ravel(), b4]).astype(np.float32)


def _samples(n, seed):
    rng = np.random.default_rng(seed)
    f = rng.uniform(-1, 1, (n, 7)).astype(np.float32)
    t = (0.1 * np.sin(2.0 * f[:, :5] + f[:, 2:7])).astype(np.float32)
    return f, t


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind in ("driver", "advance"):
        grid = _grid(c["mesh"], c["nx"], c["ny"], c["nz"])
        cfg = _config(c)
        U0 = _pinned(_initial_state(c, seed))
        s = S.EulerSolver(cfg, grid, U0=U0)
        s.tune()
        return {"kind": kind, "solver": s, "config": cfg, "U0": U0, "out": _pinned(np.zeros_like(U0)),
                "steps": c["steps"], "single": c["precision"] == "mixed32"}
    if kind == "steady":
        ch = _channels(c, seed)
        grids = [_grid("bump", k["nx"], k["nx"] // 2, k["nx"] // 2, k["h"]) for k in ch]
        batch = S.Mesh.concat(grids)
        fss = [mg.bump_freestream(k["mach"]) for k in ch]
        fs = fss[0]
        cfg = S.Config(precision="mixed", CFL=0.8, local_time_stepping=True, density_fs=fs[0],
                       velocity_fs=list(fs[1:4]), pressure_fs=fs[4], limiter="Barth" if c["ratchet"] else "NONE",
                       limiter_ratchet_step=c["ratchet"])
        U0 = _pinned(np.concatenate([mg.uniform_state(g.n_cells, f) for g, f in zip(grids, fss)]))
        s = S.EulerSolver(cfg, batch, U0=U0, patch_states=[list(f) for f, g in zip(fss, grids) for _ in g.patches()])
        s.tune()
        return {"kind": kind, "solver": s, "U0": U0, "out": _pinned(np.zeros_like(U0)), "fss": fss,
                "offsets": batch.case_offsets(), "steps": c["steps"], "check": c["check"]}
    if kind == "train":
        m = sur.MLP(seed=0)
        m.set_params(_network(seed))
        m.set_data(*_samples(c["samples"], seed))
        return {"kind": kind, "mlp": m, "batch": c["batch"], "steps": c["steps"]}
    if kind == "predict":
        m = sur.MLP(seed=0)
        m.set_params(_network(seed))
        return {"kind": kind, "mlp": m, "features": _samples(c["samples"], seed)[0]}
    if kind == "wall":
        grid = _grid("bump", c["nx"], c["ny"], c["nz"])
        export = dict(grid.export())
        # the cells of a slightly moved channel (the walls stay where they are)
        shift = np.random.default_rng(seed).uniform(-0.2, 0.2, 3) / c["nx"]
        export["centroid"] = export["centroid"] + shift
        return {"kind": kind, "grid": grid, "export": export}
    t = _tets("bump", c["nx"], c["ny"], c["nz"])
    scale = np.random.default_rng(seed).uniform(0.5, 2.0, 3)
    return {"kind": kind, "tets": mg.TetMesh(t.nodes * scale, t.tets, t.markers, t.patch_types, t.shape)}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(st):
    kind = st["kind"]
    if kind == "driver":
        s, cfg = st["solver"], st["config"]
        s.set_state(st["U0"])
        for _ in range(st["steps"]):
            s.calc_timestep(cfg)
            s.step(cfg)
        return s.get_solver_data().get_solution()
    if kind == "advance":
        s = st["solver"]
        s.upload_begin(st["U0"])
        s.upload_commit()
        s.advance(st["steps"])
        s.snapshot_begin(st["out"])
        U = s.snapshot_wait()
        # the FP32-copy form is good to single precision: its fields are kept in that
        return torch.from_numpy(U).float() if st["single"] else U
    if kind == "steady":
        s = st["solver"]
        s.upload_begin(st["U0"])
        s.upload_commit()
        res = s.solve_steady(1e-9, max_steps=st["steps"], check_every=st["check"])
        s.snapshot_begin(st["out"])
        U = s.snapshot_wait()
        off = st["offsets"]
        return {"steps": res["steps"],
                "targets": [sur.normalise_state(U[off[k]:off[k + 1]], fs) for k, fs in enumerate(st["fss"])]}
    if kind == "train":
        st["mlp"].train(st["steps"], st["batch"], 1e-3, seed=3, n_report=1)
        return st["mlp"].get_params()
    if kind == "predict":
        return st["mlp"].predict(st["features"])[0]
    if kind == "wall":
        return sur.wall_distance(st["grid"], st["export"])
    m = S.Mesh.from_tet_mesh(st["tets"], device=-1)
    return m.export()


def work(case):
    c, kind = case, case["kind"]
    if kind in ("driver", "advance", "steady"):
        if kind == "steady":
            cells = sum(6 * k["nx"] * (k["nx"] // 2) ** 2 for k in _channels(c, 0))
            second, rk3, lts, real = True, True, True, 4
        else:
            cells = 6 * c["nx"] * c["ny"] * c["nz"]
            second, rk3, lts = c["order"] == "Second", c["scheme"] == "TVD_RK3", c["lts"]
            real = 8 if c["precision"] == "fp64" else 4
        stages = 3 if rk3 else 1
        # per cell and stage: the FP64 state in and out, U^n at stages 2 and 3, four neighbours and
        # four vertices as 32-bit ids; per step the local time step out and in
        state = stages * (40 + 40 + 32) + (2 * 40 if rk3 else 0) + (16 if lts else 0)
        # per cell and stage: two face fluxes (each face shared by two cells), the reconstruction and
        # limiter of five variables, the update
        flops = stages * (2 * 130 + (5 * 30 if second else 0) + 40)
        return {"bytes": float(c["steps"]) * cells * state + 80.0 * cells, "flops": float(c["steps"]) * cells * flops}
    if kind == "train":
        return {"bytes": float(c["steps"]) * (c["batch"] * 48 + N_PARAM_USED * 24),
                "flops": 6.0 * c["steps"] * c["batch"] * N_PARAM_USED}
    if kind == "predict":
        return {"bytes": c["samples"] * 48.0, "flops": 2.0 * c["samples"] * N_PARAM_USED}
    cells = 6 * c["nx"] * c["ny"] * c["nz"]
    if kind == "wall":
        wall = 4 * c["nx"] * (c["ny"] + c["nz"])
        return {"bytes": 16.0 * cells + 12.0 * wall, "flops": 8.0 * cells * np.log2(wall)}
    return {"bytes": cells * (32.0 + 4.0 + 2 * 80.0 + 80.0), "flops": cells * 200.0}


# ---------------------------------------------------------------------------
# the same in 64 bits, from plain torch and numpy
# ---------------------------------------------------------------------------
def _conserved(V):
    U = V.clone()
    U[:, 1:4] = V[:, :1] * V[:, 1:4]
    U[:, 4] = V[:, 4] / (GAMMA - 1) + 0.5 * V[:, 0] * (V[:, 1:4] ** 2).sum(1)
    return U


def _primitive(U):
    V = U.clone()
    V[:, 1:4] = U[:, 1:4] / U[:, :1]
    V[:, 4] = (GAMMA - 1) * (U[:, 4] - 0.5 * (U[:, 1:4] ** 2).sum(1) / U[:, 0])
    return V


class _Faces:
    """Face-based grid of a tetrahedral mesh: interior faces by (i, j), then each marker's faces by
    owner; normals from i to j, vectors from the centroids to the face's centroid."""

    def __init__(self, tm):
        dev = _device()
        self.nodes = x = torch.from_numpy(tm.nodes).to(dev)
        tet = torch.from_numpy(tm.tets).to(dev)
        n, nn = tet.shape[0], x.shape[0]
        key = lambda t: (t[:, 0] * nn + t[:, 1]) * nn + t[:, 2]
        f = torch.stack([tet[:, [0, 1, 2]], tet[:, [0, 1, 3]], tet[:, [0, 2, 3]], tet[:, [1, 2, 3]]], 1).reshape(-1, 3)
        f = f.sort(1).values
        k, at = key(f).sort(stable=True)
        twin = k[1:] == k[:-1]
        a = torch.nonzero(twin).ravel()
        lo, hi = at[a] // 4, at[a + 1] // 4
        i, j = torch.minimum(lo, hi), torch.maximum(lo, hi)
        order = (i * n + j).sort().indices
        i, j, tri = i[order], j[order], f[at[a]][order]
        single = torch.ones_like(k, dtype=torch.bool)
        single[1:][twin] = False
        single[:-1][twin] = False
        kb, cb = k[single], at[single] // 4
        bi, bj, bt, self.first, ghost = [], [], [], [i.numel()], n
        for _, t in tm.markers:
            t = torch.from_numpy(t).to(dev).sort(1).values
            owner = cb[torch.searchsorted(kb, key(t))]
            o = owner.sort(stable=True).indices
            bi.append(owner[o])
            bj.append(ghost + o)
            bt.append(t[o])
            ghost += t.shape[0]
            self.first.append(self.first[-1] + t.shape[0])
        self.n, self.ni = n, i.numel()
        self.i, self.j = torch.cat([i] + bi), torch.cat([j] + bj)
        tri = torch.cat([tri] + bt)
        p, q, r = (x[tri[:, v]] for v in range(3))
        fc = (p + q + r) / 3
        t0, t1, t2, t3 = (x[tet[:, v]] for v in range(4))
        cen = (t0 + t1 + t2 + t3) / 4
        self.vol = (torch.linalg.cross(t1 - t0, t2 - t0) * (t3 - t0)).sum(1).abs() / 6
        self.centroid = torch.cat([cen, torch.empty(ghost - n, 3, dtype=cen.dtype, device=dev)])
        b = slice(self.ni, None)
        self.centroid[self.j[b]] = 2 * fc[b] - cen[self.i[b]]
        S_ = 0.5 * torch.linalg.cross(q - p, r - p)
        self.ri, self.rj = fc - self.centroid[self.i], fc - self.centroid[self.j]
        self.S = torch.where(((self.centroid[self.j] - self.centroid[self.i]) * S_).sum(1, keepdim=True) < 0, -S_, S_)
        half = 0.5 * self.S[:self.ni].abs()
        self.dS = torch.zeros(n, 3, dtype=cen.dtype, device=dev)
        self.dS.index_add_(0, self.i[:self.ni], half)
        self.dS.index_add_(0, self.j[:self.ni], half)


def _ghost(kind, fs, V, n, density_fix):
    G = V.clone()
    vn = (V[:, 1:4] * n).sum(1, keepdim=True)
    if kind == mg.SLIP_WALL:
        G[:, 1:4] = V[:, 1:4] - 2 * vn * n
        return G
    rho, v, p = fs[0], torch.tensor(fs[1:4], dtype=V.dtype, device=V.device), fs[4]
    g1, c_fs = GAMMA - 1, (GAMMA * p / rho) ** 0.5
    vn_fs, vn = (n * v).sum(1), vn[:, 0]
    c = torch.sqrt(GAMMA * V[:, 4] / V[:, 0])
    Rp = torch.where(vn_fs + c_fs > 0, vn + 2 * c / g1, vn_fs + 2 * c_fs / g1)
    Rm = torch.where(vn_fs - c_fs > 0, vn - 2 * c / g1, vn_fs - 2 * c_fs / g1)
    vb, cb = 0.5 * (Rp + Rm), g1 / 4 * (Rp - Rm)
    out = (vn_fs > 0)[:, None]
    G[:, 1:4] = torch.where(out, V[:, 1:4] + (vb - vn)[:, None] * n, v + (vn_fs - vb)[:, None] * n)
    s = torch.where(out[:, 0], V[:, 4] * V[:, 0] ** -GAMMA, torch.full_like(vn, p * rho ** -GAMMA))
    ratio = cb * cb / (GAMMA * s) if density_fix else GAMMA * s / (cb * cb)
    G[:, 0] = ratio ** (1 / g1)
    G[:, 4] = cb * cb * G[:, 0] / GAMMA
    return G


def _march(tm, U0, fs, steps, lts, second, rk3, barth, ratchet=0, patch_fs=None, density_fix=False):
    """steps x (time step from the last stage's primitives, step): Green-Gauss gradients, the Barth
    limiter, Rusanov fluxes, explicit Euler or TVD-RK3; the ratchet keeps the limiter's minimum."""
    g = _Faces(tm)
    n, ni, i, j = g.n, g.ni, g.i, g.j
    U = torch.from_numpy(np.ascontiguousarray(U0)).to(g.vol.device)
    area = g.S.norm(dim=1, keepdim=True)
    nrm = g.S / area
    ji, eps = j[:ni], np.finfo(np.float64).eps
    vol = g.vol[:, None]
    patches = [(slice(g.first[k], g.first[k + 1]), tm.patch_types[name], (patch_fs or {}).get(name, fs))
               for k, (name, _) in enumerate(tm.markers)]
    kept = None

    def ghosts(Vb):
        return torch.cat([_ghost(t, f, Vb[s.start - ni:s.stop - ni], nrm[s], density_fix) for s, t, f in patches])

    def flux(L, R):
        def side(V):
            vn = (V[:, 1:4] * nrm).sum(1, keepdim=True)
            W = _conserved(V)
            F = W * vn
            F[:, 1:4] += V[:, 4:] * nrm
            F[:, 4:] += V[:, 4:] * vn
            return W, F, vn.abs() + torch.sqrt(GAMMA * V[:, 4:] / V[:, :1])
        (UL, FL, sL), (UR, FR, sR) = side(L), side(R)
        return 0.5 * area * (FL + FR - torch.maximum(sL, sR) * (UR - UL))

    def scatter(t):  # sum over a cell's faces, the owner's sign +
        out = torch.zeros(n, t.shape[1], dtype=t.dtype, device=t.device)
        out.index_add_(0, i, t)
        out.index_add_(0, ji, t[:ni], alpha=-1)
        return out

    def balance(U, step):
        nonlocal kept
        V = _primitive(U)
        Vi = V[i]
        Vj = torch.cat([V[ji], ghosts(Vi[ni:])])
        L, R = Vi, Vj
        if second:
            mean = 0.5 * (Vi + Vj)
            grad = torch.stack([scatter(mean * g.S[:, d:d + 1]) / vol for d in range(3)])  # [3][n][5]
            at = lambda c, r: sum(grad[d][c] * r[:, d:d + 1] for d in range(3))
            di, dj = at(i, g.ri), at(ji, g.rj[:ni])
            phi = torch.ones_like(V)
            if barth:
                idx_i, idx_j = i[:, None].expand(-1, 5), ji[:, None].expand(-1, 5)
                both = lambda op, lim: (lim.scatter_reduce_(0, idx_i, op(Vi, Vj), "amax" if op is torch.maximum else "amin"),
                                        lim.scatter_reduce_(0, idx_j, op(Vi, Vj)[:ni], "amax" if op is torch.maximum else "amin"))[1]
                hi, lo = both(torch.maximum, V.clone()), both(torch.minimum, V.clone())

                def ratio(c, d):
                    room = torch.where(d > 0, hi[c] - V[c], lo[c] - V[c])
                    return torch.where(d == 0, 1.0, torch.clamp(room / (d + torch.sign(d) * eps), max=1.0))
                phi.scatter_reduce_(0, idx_i, ratio(i, di), "amin")
                phi.scatter_reduce_(0, idx_j, ratio(ji, dj), "amin")
                if ratchet and step >= ratchet:
                    kept = phi if kept is None else torch.minimum(kept, phi)
                    phi = kept
            L = Vi + phi[i] * di
            R = torch.cat([Vj[:ni] + phi[ji] * dj, ghosts(L[ni:])])
        return V, -scatter(flux(L, R))

    def time_step(V):
        c = torch.sqrt(GAMMA * V[:, 4:] / V[:, :1])
        dt = 0.8 * g.vol / ((V[:, 1:4].abs() + c) * g.dS).sum(1)
        return (dt if lts else dt.min()[None])[:, None] / vol
    V = _primitive(U)
    for step in range(steps):
        q, Un = time_step(V), U
        V, R = balance(U, step)
        U = Un + q * R
        if rk3:
            V, R = balance(U, step)
            U = 0.75 * Un + 0.25 * U + 0.25 * q * R
            V, R = balance(U, step)
            U = Un / 3 + 2 * U / 3 + 2 / 3 * q * R
    return U


def _layers(p):
    """Weights and biases in 64 bits from the parameter vector (W0's column 7 is its bias)."""
    p = torch.from_numpy(p).to(_device()).double()
    W0, W = p[:2048].view(128, 16), p[2048:2048 + 49152].view(3, 128, 128)
    b, W4, b4 = p[51200:51584].view(3, 128), p[51584:53632].view(16, 128), p[53632:53648]
    return [W0[:, :7].clone(), W[0].clone(), W[1].clone(), W[2].clone(), W4[:5].clone()], \
           [W0[:, 7].clone(), b[0].clone(), b[1].clone(), b[2].clone(), b4[:5].clone()]


def _flat(W, b):
    out = torch.zeros(53648, dtype=torch.float64, device=W[0].device)
    W0, W4 = out[:2048].view(128, 16), out[51584:53632].view(16, 128)
    W0[:, :7], W0[:, 7], W4[:5] = W[0], b[0], W[4]
    out[2048:51200] = torch.stack(W[1:4]).ravel()
    out[51200:51584] = torch.stack(b[1:4]).ravel()
    out[53632:53637] = b[4]
    return out


def _forward(W, b, x):
    for k in range(4):
        x = torch.nn.functional.silu(x @ W[k].T + b[k])
    return x @ W[4].T + b[4]


def _batch(step, batch, n, seed):
    """The sampled rows of a training step: splitmix64 of a running counter, modulo the sample count."""
    with np.errstate(over="ignore"):
        z = np.arange(1, batch + 1, dtype=np.uint64) + np.uint64(step) * np.uint64(batch)
        z = z * np.uint64(0x9E3779B97F4A7C15) + np.uint64(seed)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z ^= z >> np.uint64(31)
    return (z % np.uint64(n)).astype(np.int64)


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("driver", "advance"):
        cfg = {"patch_fs": {"left": mg.SOD_LEFT, "right": mg.SOD_RIGHT}, "density_fix": True} \
            if c["mesh"] == "sod" else {}
        return _march(_tets(c["mesh"], c["nx"], c["ny"], c["nz"]), _initial_state(c, seed), _freestream(c),
                      c["steps"], c["lts"], c["order"] == "Second", c["scheme"] == "TVD_RK3",
                      c["limiter"] == "Barth" and c["order"] == "Second", **cfg)
    if kind == "steady":
        targets, n = [], 0
        for k in _channels(c, seed):
            tm = _tets("bump", k["nx"], k["nx"] // 2, k["nx"] // 2, k["h"])
            rho, u, v, w, p = fs = mg.bump_freestream(k["mach"])
            U = _march(tm, mg.uniform_state(tm.n_cells, fs), fs, c["steps"], True, True, True, c["ratchet"] > 0,
                       c["ratchet"])
            speed = (u * u + v * v + w * w) ** 0.5
            E = p / (GAMMA - 1) + 0.5 * rho * speed * speed
            scale = torch.tensor([rho, rho * speed, rho * speed, rho * speed, E], dtype=U.dtype, device=U.device)
            base = torch.tensor([1, u / speed, v / speed, w / speed, 1], dtype=U.dtype, device=U.device)
            targets.append(U / scale - base)
            n += 1
        return {"steps": np.full(n, c["steps"], np.int64), "targets": targets}
    if kind == "train":
        W, b = _layers(_network(seed))
        f, t = (torch.from_numpy(a).to(W[0].device).double() for a in _samples(c["samples"], seed))
        par = W + b
        mom = [(torch.zeros_like(p), torch.zeros_like(p)) for p in par]
        for step in range(1, c["steps"] + 1):
            at = torch.from_numpy(_batch(step, c["batch"], c["samples"], 3)).to(f.device)
            leaf = [p.clone().requires_grad_() for p in par]
            ((_forward(leaf[:5], leaf[5:], f[at]) - t[at]) ** 2).mean().backward()
            for p, q, (m, v) in zip(par, leaf, mom):
                m.mul_(0.9).add_(q.grad, alpha=0.1)
                v.mul_(0.999).addcmul_(q.grad, q.grad, value=0.001)
                p -= 1e-3 * (m / (1 - 0.9 ** step)) / (torch.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
        return _flat(par[:5], par[5:])
    if kind == "predict":
        W, b = _layers(_network(seed))
        x = torch.from_numpy(_samples(c["samples"], seed)[0]).to(W[0].device).double()
        return torch.cat([_forward(W, b, p) for p in x.split(250000)])
    if kind == "wall":
        g = _Faces(_tets("bump", c["nx"], c["ny"], c["nz"]))
        tm = _tets("bump", c["nx"], c["ny"], c["nz"])
        shift = torch.from_numpy(np.random.default_rng(seed).uniform(-0.2, 0.2, 3) / c["nx"]).to(g.vol.device)
        x = g.centroid[:g.n] + shift
        walls = [slice(g.first[k], g.first[k + 1]) for k, (name, _) in enumerate(tm.markers)
                 if tm.patch_types[name] == mg.SLIP_WALL]
        w = torch.cat([x[g.i[s]] + g.ri[s] for s in walls])
        chunk = max(1, 100_000_000 // w.shape[0])
        return torch.cat([torch.cdist(p, w, compute_mode="donot_use_mm_for_euclid_dist").min(1).values
                          for p in x.split(chunk)])
    t = _tets("bump", c["nx"], c["ny"], c["nz"])
    scale = np.random.default_rng(seed).uniform(0.5, 2.0, 3)
    g = _Faces(mg.TetMesh(t.nodes * scale, t.tets, t.markers, t.patch_types, t.shape))
    n_all = g.centroid.shape[0]
    vol = torch.zeros(n_all, dtype=g.vol.dtype, device=g.vol.device)
    vol[:g.n] = g.vol
    return {"face_ij": torch.stack([g.i, g.j], 1), "S": g.S, "ri": g.ri, "rj": g.rj, "vol": vol,
            "centroid": g.centroid, "dS": g.dS}
