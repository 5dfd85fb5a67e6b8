"""The work that a user of this framework has it do, as measurable cases.

Every case is one whole call sequence of a user's program: the state of a
community (or medium, or rod colony) goes in from host arrays, the framework
advances it, and the new state comes back to host arrays (loadToPlatform!,
step! x n, bringFromPlatform!), or one call that does the three by itself
(the adjoint).  Agent communities go through the C ABI on host buffers laid
out once, as the Julia binding calls it; the other parts through the package's
classes.

Families, and what each stands for:
  aggregation  small soft-sphere tissue, Euler, reflecting walls: the tutorial
               size, where launches and latency count
  colony       the growing 3D colony (division, death, Euler-Maruyama, CLVD):
               young (1e4, loose) to grown (1e6, about 350 neighbors an agent)
  tissue       a fixed 3D community on Verlet lists (CLVD), rebuilt on displacement
  chemotaxis   2D agents coupled to an FTCS medium (secretion, gradient drift)
  medium3d     the same coupling in 3D with uptake; the field dominates
  sweep        many independent communities of uneven sizes in one batch
  adjoint      forward and backward through a trajectory
  dgadi        implicit (Douglas-Gunn ADI) medium, 2D and 3D
  rods         2D rod colony, with and without growth

`exact` restates each family in Float64 with torch alone.  Where agents are
born and die, the community's size depends on comparisons of rounded volumes
(which agents divide in which step), so a colony has no such value; nor have
the chemotaxis agents, whose step amplifies every rounding.
"""
import ctypes as C
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    if "cbm_b200" not in sys.modules:
        pkg = os.path.join(ROOT, "cellbasedmodels.jl_b200")
        spec = importlib.util.spec_from_file_location(
            "cbm_b200", os.path.join(pkg, "__init__.py"), submodule_search_locations=[pkg])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["cbm_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["cbm_b200"]


def listed():
    return [
        # a tutorial-size tissue followed closely: few agents, few steps a call
        dict(name="aggregation_small", family="aggregation", dims=2, n=700, steps=20, dtype="f64",
             neighbors="cell"),
        # the 2D aggregation at its documented size, Float64 as the reference runs it
        dict(name="aggregation_4096", family="aggregation", dims=2, n=4096, steps=200,
             dtype="f64", neighbors="cell"),
        # the growing colony at its start: loose, latency-bound
        dict(name="colony_young", family="colony", n=10_000, steps=100, dtype="f32"),
        # the colony half grown, in Float64
        dict(name="colony_f64", family="colony", n=150_001, steps=20, dtype="f64"),
        # the colony grown to 10^6
        dict(name="colony_grown", family="colony", n=1_000_000, steps=8, dtype="f32"),
        # a confluent tissue without births, stepped on its Verlet lists
        dict(name="tissue_lists", family="tissue", n=100_003, steps=60, dtype="f32", skin=0.6),
        # chemotaxis on a 1024^2 medium between two saves
        dict(name="chemotaxis", family="chemotaxis", n=200_000, nodes=1024, steps=100,
             dtype="f32"),
        # a 3D medium with its agents between two saves
        dict(name="medium_3d", family="medium3d", n=200_000, nodes=256, steps=100, dtype="f32"),
        # one generation of a parameter fit: 512 communities
        dict(name="sweep_512", family="sweep", communities=512, n_lo=500, n_hi=20_000, steps=50),
        # gradients of a trajectory loss
        dict(name="adjoint", family="adjoint", n=65_536, steps=100, every=20, dtype="f64"),
        # the implicit medium of the reference's notebook, 3D
        dict(name="dgadi_3d", family="dgadi", dims=3, nodes=101, fields=2, steps=100,
             dtype="f32"),
        # a rod colony of the reference's notebook
        dict(name="rods", family="rods", n=32_768, steps=100, dtype="f64", growth=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    fam = rng.choice(["aggregation", "colony", "colony", "tissue", "chemotaxis", "medium3d",
                      "sweep", "adjoint", "dgadi", "rods"])
    dtype = rng.choice(["f32", "f64"])
    if fam == "aggregation":
        alg = rng.choice(["cell", "cell", "verlet", "full"])
        return dict(family=fam, dims=rng.choice([2, 3]),
                    n=_log(rng, 300, 30_000 if alg == "cell" else 5_000),
                    steps=rng.randint(10, 200), dtype=dtype, neighbors=alg)
    if fam == "colony":
        n = _log(rng, 5_000, 1_000_000 if dtype == "f32" else 300_000)
        return dict(family=fam, n=n, steps=max(4, min(100, 6_000_000 // n)), dtype=dtype)
    if fam == "tissue":
        return dict(family=fam, n=_log(rng, 2_000, 300_000), steps=rng.randint(20, 60),
                    dtype=dtype, skin=rng.choice([0.3, 0.6, 1.0]))
    if fam == "chemotaxis":
        m = _log(rng, 120, 1024)
        return dict(family=fam, n=max(200, int(m * m * rng.uniform(0.05, 0.19))), nodes=m,
                    steps=rng.randint(20, 100), dtype=dtype)
    if fam == "medium3d":
        m = _log(rng, 40, 256 if dtype == "f32" else 200)
        return dict(family=fam, n=max(500, int(m ** 3 * rng.uniform(0.003, 0.012))), nodes=m,
                    steps=rng.randint(20, 100), dtype=dtype)
    if fam == "sweep":
        hi = _log(rng, 1_000, 20_000)
        return dict(family=fam, communities=_log(rng, 16, 512), n_lo=max(300, hi // 20), n_hi=hi,
                    steps=rng.randint(20, 50))
    if fam == "adjoint":
        return dict(family=fam, n=_log(rng, 1_500, 65_536), steps=rng.randint(20, 100),
                    every=rng.choice([5, 10, 20]), dtype=rng.choice(["f64", "f64", "f32"]))
    if fam == "dgadi":
        dims = rng.choice([2, 3])
        return dict(family=fam, dims=dims, nodes=_log(rng, 20, 400 if dims == 2 else 110),
                    fields=rng.randint(1, 2), steps=rng.randint(20, 100), dtype=dtype)
    return dict(family=fam, n=_log(rng, 800, 32_768), steps=rng.randint(20, 100), dtype=dtype,
                growth=rng.choice([False, True]))


# ---- inputs -------------------------------------------------------------------
def _np(case):
    return np.float64 if case.get("dtype") == "f64" else np.float32


def _ball(rng, n):
    """A colony of n agents: the radial density of the grown colony (about
    4.7 sqrt(n / 1e6) agents per unit volume in its core, thinning outwards)."""
    core = max(0.3, 4.7 * math.sqrt(n / 1e6))
    s = np.linspace(0, 1, 201)
    rho = np.interp(s, [0, 0.35, 0.75, 0.85, 1.0], [1, 0.97, 0.68, 0.45, 0.03])
    cdf = np.concatenate([[0], np.cumsum((rho[1:] + rho[:-1]) / 2 * np.diff(s ** 3))])
    R = (3 * n / (4 * math.pi * core * cdf[-1])) ** (1 / 3)
    r = R * np.interp(rng.random(n), cdf / cdf[-1], s)
    u = rng.normal(size=(3, n))
    u /= np.linalg.norm(u, axis=0)
    return 200.0 + u * r


def _setup(case, seed):
    """(configuration keywords, host state) of an agent community."""
    abi = _package()._abi
    fam, n, dt_ = case["family"], case["n"], _np(case)
    rng = np.random.default_rng([seed, n])
    kw = dict(precision=abi.F64 if dt_ == np.float64 else abi.F32, seed=seed, n_max=n,
              k_rep=10.0, r_rep=2.0)
    if fam == "aggregation":
        D = case["dims"]
        L = 100.0 * math.sqrt(n / 4096) if D == 2 else 2.5 * n ** (1 / 3)
        alg = dict(cell=abi.NEIGH_CELL_LINKED, verlet=abi.NEIGH_VERLET_DISPLACEMENT,
                   full=abi.NEIGH_FULL)[case["neighbors"]]
        kw.update(dims=D, box_lo=(0.0,) * D, box_hi=(L,) * D, dt=0.01, neighbors=alg,
                  cell_edge=3.0, skin=3.6, n_max_neighbors=256, integrator=abi.INT_EULER,
                  k_att=1.0, r_att=3.0, walls=abi.WALLS_REFLECT)
        pos = rng.uniform(0, L, (D, n))
    elif fam == "colony":
        kw.update(dims=3, n_max=int(n * (1 + 0.008 * case["steps"])) + 1000, box_lo=(0.0,) * 3,
                  box_hi=(400.0,) * 3, dt=0.005, neighbors=abi.NEIGH_CLVD, cell_edge=3.3, skin=3.3,
                  rebuild_threshold=0.15, n_max_neighbors=1024, integrator=abi.INT_EM, sigma=0.05,
                  k_att=1.0, r_att=3.0, growth=1, fate=abi.FATE_VOLUME, v_div=2.0, div_sep=0.5,
                  p_death=1e-4)
        pos = _ball(rng, n)
    elif fam == "tissue":
        L, R = 2.5 * n ** (1 / 3), 3.0 + case["skin"]
        kw.update(dims=3, box_lo=(0.0,) * 3, box_hi=(L,) * 3, dt=0.01, neighbors=abi.NEIGH_CLVD,
                  cell_edge=R, skin=R, rebuild_threshold=case["skin"] / 2, n_max_neighbors=256,
                  integrator=abi.INT_EM, sigma=0.05, k_att=1.0, r_att=3.0)
        pos = rng.uniform(0, L, (3, n))
    elif fam == "chemotaxis":
        L = float(case["nodes"])
        kw.update(dims=2, box_lo=(0.0,) * 2, box_hi=(L,) * 2, dt=0.2,
                  neighbors=abi.NEIGH_CELL_LINKED, cell_edge=2.0, integrator=abi.INT_EM,
                  sigma=0.1, k_att=0.0, r_att=2.0, medium=1, n_medium=(case["nodes"],) * 2,
                  diff_D=1.0, decay=0.01, secretion=0.1, chemotaxis=0.5,
                  medium_sampling=abi.MEDIUM_BILINEAR)
        pos = rng.uniform(0, L, (2, n))
    else:
        L = float(case["nodes"])
        kw.update(dims=3, box_lo=(0.0,) * 3, box_hi=(L,) * 3, dt=0.05,
                  neighbors=abi.NEIGH_CELL_LINKED, cell_edge=2.4, integrator=abi.INT_EM,
                  sigma=0.1, k_att=0.0, r_att=2.0, medium=1, n_medium=(case["nodes"],) * 3,
                  diff_D=1.0, decay=0.01, secretion=0.1, uptake=0.05, chemotaxis=0.5,
                  medium_sampling=abi.MEDIUM_BILINEAR)
        pos = rng.uniform(0, L, (3, n))
    st = {k: pos[d].astype(dt_) for d, k in enumerate("xyz"[: kw["dims"]])}
    if fam == "colony":
        st["v"] = rng.uniform(1, 2, n).astype(dt_)
        st["g"] = rng.uniform(0.8, 1.2, n).astype(dt_)
    if "nodes" in case:
        st["c"] = rng.random(case["nodes"] ** kw["dims"], dtype=np.float32).astype(dt_)
    return kw, st


def _rod_state(case, seed):
    n, dt_ = case["n"], _np(case)
    rng = np.random.default_rng([seed, n])
    r = math.sqrt(n * 3.8 / math.pi) * np.sqrt(rng.random(n))
    phi = rng.uniform(0, 2 * math.pi, n)
    st = {k: np.zeros(n) for k in _package()._abi.ROD_FIELDS}
    st["x"], st["y"] = r * np.cos(phi), r * np.sin(phi)
    st["vx"], st["vy"] = rng.normal(0, 0.01, n), rng.normal(0, 0.01, n)
    st["theta"], st["omega"] = rng.uniform(-math.pi, math.pi, n), rng.normal(0, 0.01, n)
    st["d"], st["m"], st["l"] = np.ones(n), np.ones(n), rng.uniform(2.0, 3.0, n)
    st["l_target"] = st["l"] + rng.uniform(0.0, 0.02, n)
    return {k: v.astype(dt_) for k, v in st.items()}


# the constants of the rod model's example (m = 1/100, g = 1/10000, d = 1)
_ROD = dict(dt=0.1, kn=2.0, gamma_n=2.2, gamma_t=2.2, mu_cc=0.1, mu_cw=0.8, beta=0.8, beta_w=0.8)
_ROD_GROWTH = dict(growth=1e-3, alpha=50.0, sigma_l_target=0.2, l_max=3.0)


def _sweep_setup(case, seed):
    sizes = np.random.default_rng([case["communities"], case["n_hi"]]).integers(
        case["n_lo"], case["n_hi"] + 1, case["communities"])
    rng = np.random.default_rng([seed, case["communities"]])
    descs, states = [], []
    for c, n in enumerate(int(v) for v in sizes):
        L = 2.5 * n ** (1 / 3)
        f = np.exp(rng.uniform(math.log(0.3), math.log(3.0), 3))
        descs.append(dict(n=n, L=L, k_rep=10.0 * f[0], k_att=f[1], sigma=0.05 * f[2], community=c))
        states.append((rng.random((3, n), dtype=np.float32) * np.float32(L)))
    return descs, states


def _adjoint_setup(case, seed):
    n = case["n"]
    L = 80.0 * (n / 65_536) ** (1 / 3)
    rng = np.random.default_rng([seed, n])
    x0 = rng.uniform(0, L, (3, n)).astype(_np(case))
    target = (x0 + rng.normal(0, 0.3, (3, n))).astype(_np(case))
    return L, x0, target


def _dgadi_setup(case, seed):
    D, m = case["dims"], case["nodes"]
    rng = np.random.default_rng([seed, m])
    u = rng.random((case["fields"],) + (m,) * D).astype(_np(case))
    src = np.zeros((m,) * D, _np(case))
    src[(round(m / 2) - 1,) * D] = 1.0
    return u, src, [1.0, 2.0][: case["fields"]]


def prepare(case, seed):
    cbm = _package()
    abi, fam = cbm._abi, case["family"]
    s = dict(case=case)
    if fam == "sweep":
        descs, states = _sweep_setup(case, seed)
        base = abi.make_config(dims=3, precision=abi.F32, n_max=1, dt=0.01, seed=seed,
                               neighbors=abi.NEIGH_CLVD, integrator=abi.INT_EM,
                               n_max_neighbors=256, skin=4.0, cell_edge=4.0,
                               rebuild_threshold=0.5, k_rep=10.0, r_rep=2.0, k_att=1.0, r_att=3.0)
        out = []
        for d in descs:
            x = abi.CbmCommunityDesc()
            x.n, x.box_hi = d["n"], type(x.box_hi)(*(d["L"],) * 3)
            x.r_rep, x.r_att = 2.0, 3.0
            for k in ("k_rep", "k_att", "sigma", "community"):
                setattr(x, k, d[k])
            out.append(x)
        s["batch"] = cbm.Batch(base, out)
        # the tuning that the autotuner picks for the 512-community sweep
        s["batch"].set_tuning(threads=1024, ctas_per_sm=1, skin=1.0)
        s["states"] = states
    elif fam == "adjoint":
        L, x0, target = _adjoint_setup(case, seed)
        cfg = abi.make_config(dims=3, precision=abi.F64 if case["dtype"] == "f64" else abi.F32,
                              n_max=case["n"], box_hi=(L,) * 3, dt=0.01, seed=seed,
                              neighbors=abi.NEIGH_CELL_LINKED, cell_edge=3.3,
                              integrator=abi.INT_EULER, k_rep=10.0, r_rep=2.0, k_att=1.0,
                              r_att=3.0)
        s.update(adjoint=cbm.Adjoint(cfg), x0=list(x0), target=list(target))
    elif fam == "dgadi":
        u, src, diff = _dgadi_setup(case, seed)
        D = case["dims"]
        cfg = abi.make_medium_config(D, (case["nodes"],) * D, (0.0,) * D, (1.0,) * D, 0.01, diff,
                                     c_max=1.0,
                                     precision=abi.F64 if case["dtype"] == "f64" else abi.F32)
        s.update(medium=cbm.DGADIMedium(cfg), u=u, src=src)
    elif fam == "rods":
        half = 1.2 * math.sqrt(case["n"] * 3.8 / math.pi)
        more = dict(_ROD_GROWTH, seed=seed) if case["growth"] else {}
        cfg = abi.make_rods_config(case["n"] * (2 if case["growth"] else 1), (-half,) * 2,
                                   (half,) * 2, cell_edge=4.0, neighbors=abi.NEIGH_CELL_LINKED,
                                   precision=abi.F64 if case["dtype"] == "f64" else abi.F32,
                                   **_ROD, **more)
        s.update(rods=cbm.Rods2D(cfg), state=_rod_state(case, seed))
    else:
        kw, st = _setup(case, seed)
        ctx = cbm.Context(abi.make_config(**kw))
        # host buffers in page-locked memory, one set for what goes in and one
        # for what comes back, with the C structures that point at them
        names = ["x", "y", "z"][: kw["dims"]]
        if fam == "colony":
            names += ["v", "g", "id", "parent"]
        if "nodes" in case:
            names += ["c"] + ["gx", "gy", "gz"][: kw["dims"]]
        tdt = torch.float64 if case["dtype"] == "f64" else torch.float32

        def buffers(keys):
            b = abi.StateBuffers.__new__(abi.StateBuffers)
            b.cfg, b.capacity, b.n_nodes, b.arrays = ctx.cfg, int(kw["n_max"]), ctx.n_nodes, {}
            for k in abi.StateBuffers.AGENT_REAL + abi.StateBuffers.MEDIUM + ("id", "parent"):
                if k in keys:
                    size = ctx.n_nodes if k in abi.StateBuffers.MEDIUM else b.capacity
                    kind = torch.int64 if k in ("id", "parent") else tdt
                    b.arrays[k] = torch.zeros(size, dtype=kind, pin_memory=True).numpy()
                else:
                    b.arrays[k] = None
            return b

        src, dst = buffers(st), buffers(names)
        for k, v in st.items():
            src.arrays[k][: len(v)] = v
        s.update(ctx=ctx, names=names, src=src, dst=dst, steps=case["steps"],
                 into=src.view(N=case["n"], id_max=0, fields=list(st)), back=dst.view(fields=names),
                 flags=(abi.SYNC, abi.VIEW_COMMITTED))
    return s


def run(s):
    case = s["case"]
    fam = case["family"]
    if fam == "sweep":
        b = s["batch"]
        for c, p in enumerate(s["states"]):
            b.upload(c, p[0], p[1], p[2])
        b.step(case["steps"])
        got = [b.download(c) for c in range(case["communities"])]
        return {k: np.concatenate([g[k] for g in got]) for k in "xyz"}
    if fam == "adjoint":
        return s["adjoint"].run(s["x0"], s["target"], case["steps"],
                                checkpoint_every=case["every"])
    if fam == "dgadi":
        s["medium"].upload(s["u"], s["src"])
        s["medium"].step(case["steps"])
        return s["medium"].download()[0]
    if fam == "rods":
        s["rods"].upload(s["state"])
        s["rods"].step(case["steps"])
        out = s["rods"].download()
        rows = s["rods"].cfg.n_max  # a growing colony's rows beyond its count stay zero
        return {k: np.pad(v, (0, rows - len(v))) for k, v in out.items()} if case["growth"] else out
    ctx, back = s["ctx"], s["back"]
    sync, committed = s["flags"]
    ctx._check(ctx.lib.cbm_upload(ctx.h, C.byref(s["into"])))
    ctx._check(ctx.lib.cbm_step(ctx.h, s["steps"], sync))
    back.capacity = s["dst"].capacity
    ctx._check(ctx.lib.cbm_download(ctx.h, C.byref(back), committed))
    # a colony's buffers hold its capacity: the first N rows are the agents
    return {k: s["dst"].arrays[k] for k in s["names"]} | {"N": int(back.N)}


def work(case):
    """One pass: every step reads and writes the state it advances; an agent's
    pair terms cost about 20 operations each."""
    fam, steps = case["family"], case["steps"]
    s = 8 if case.get("dtype") == "f64" else 4
    if fam == "sweep":
        n = case["communities"] * (case["n_lo"] + case["n_hi"]) // 2
        return dict(bytes=steps * n * 24, flops=steps * n * 7.2 * 20)
    n = case.get("n", 0)
    if fam == "adjoint":  # forward and backward: positions and their adjoints, 14.5 partners
        return dict(bytes=steps * n * 12 * s, flops=steps * n * 14.5 * 70)
    if fam == "dgadi":  # a tridiagonal solve per axis: 8 operations a node
        nodes = case["fields"] * case["nodes"] ** case["dims"]
        return dict(bytes=steps * nodes * 2 * s, flops=steps * nodes * (3 + 8 * case["dims"]))
    if fam == "rods":  # 38 candidates a rod, about 80 operations to decide on each
        return dict(bytes=steps * n * 21 * s, flops=steps * n * 38 * 80)
    if fam == "colony":
        near = 113.0 * 0.75 * max(0.3, 4.7 * math.sqrt(n / 1e6))
        return dict(bytes=steps * n * 9 * s, flops=steps * n * (near * 20 + 100))
    if fam == "tissue":
        return dict(bytes=steps * n * 6 * s, flops=steps * n * (7.2 * 20 + 100))
    if fam == "aggregation":
        D = case["dims"]
        near = 11.6 if D == 2 else 7.2
        return dict(bytes=steps * n * 2 * D * s, flops=steps * n * near * 20)
    D = 2 if fam == "chemotaxis" else 3
    nodes = case["nodes"] ** D
    return dict(bytes=steps * (nodes * 2 + n * 2 * D) * s,
                flops=steps * (nodes * (3 + 4 * D) + n * 300))


# ---- the same in Float64, with torch alone --------------------------------------
_DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.asarray(a, np.float64), device=_DEV)


class _Grid:
    """The cells of one or more communities: edge `edge`, a ghost layer around
    each box [0, hi], and everything beyond a box in its outermost cells.  With
    `wide` the cells go on beyond the box instead (all pairs are found)."""

    def __init__(self, D, hi, edge, own, wide=False):
        self.D, self.edge, self.own = D, edge, own
        self.hi = torch.as_tensor(hi, dtype=torch.float64, device=_DEV).reshape(-1, 1).repeat(1, D)
        self.pad = 40 if wide else 1
        self.wide = wide
        self.nc = torch.ceil(self.hi / edge).long() + 2 * self.pad
        total = self.nc.prod(1)
        self.base, self.total = torch.cumsum(total, 0) - total, int(total.sum())

    def cells(self, x):
        hi, nc = self.hi[self.own].T, self.nc[self.own].T
        q = torch.clamp(torch.floor(x / self.edge).long() + self.pad, min=0)
        q = torch.minimum(q, nc - 1)
        return q if self.wide else torch.where(x > hi, nc - 1, torch.where(x >= 0, q, 0))

    def pairs(self, x, x_grid, among=None):
        """(i, j), i != j: j (of those in `among`) filed by x_grid in a cell next
        to the cell of x_i."""
        D, nc = self.D, self.nc[self.own].T
        me = torch.arange(x.shape[1], device=x.device) if among is None else among
        nc, base = nc[:, me], self.base[self.own[me]]

        def linear(q):
            lin = q[0]
            for d in range(1, D):
                lin = lin + q[d] * nc[:d].prod(0)
            return lin + base

        filed = linear(self.cells(x_grid)[:, me])
        order = torch.argsort(filed, stable=True)
        start = torch.searchsorted(filed[order], torch.arange(self.total + 1, device=x.device))
        q = self.cells(x)[:, me]
        ii, jj = [], []
        for dz in (-1, 0, 1) if D > 2 else (0,):
            for dy in (-1, 0, 1) if D > 1 else (0,):
                ok = torch.ones(len(me), dtype=torch.bool, device=x.device)
                row = [torch.zeros_like(q[0])] + [q[d] + (dy, dz)[d - 1] for d in range(1, D)]
                for d in range(1, D):
                    ok &= (row[d] >= 0) & (row[d] < nc[d])
                row = torch.where(ok, linear(row), 0)
                a = start[row + torch.where(ok, torch.clamp(q[0] - 1, min=0), 0)]
                b = start[row + torch.where(ok, torch.minimum(q[0] + 1, nc[0] - 1), 0) + 1]
                cnt = torch.where(ok, b - a, 0)
                i = torch.repeat_interleave(torch.arange(len(me), device=x.device), cnt)
                first = torch.cumsum(cnt, 0) - cnt
                j = order[a[i] + torch.arange(len(i), device=x.device) - first[i]]
                keep = i != j
                ii.append(me[i[keep]])
                jj.append(me[j[keep]])
        return torch.cat(ii), torch.cat(jj)


class _Lists:
    """Verlet lists of radius R over a grid, made anew for a community when one
    of its agents has moved by `threshold`."""

    def __init__(self, grid, R, threshold, x):
        self.grid, self.R, self.threshold = grid, R, threshold
        self.i = self.j = torch.zeros(0, dtype=torch.long, device=x.device)
        self.old = torch.full_like(x, math.inf)
        self.check(x)

    def check(self, x):
        own = self.grid.own
        moved = ~(((x - self.old) ** 2).sum(0) < self.threshold ** 2)
        flag = torch.zeros(len(self.grid.hi), dtype=torch.bool, device=x.device)
        flag[own[moved]] = True
        if not bool(flag.any()):
            return
        on = flag[own]
        i, j = self.grid.pairs(x, x, torch.nonzero(on).reshape(-1))
        near = ((x[:, i] - x[:, j]) ** 2).sum(0) < self.R ** 2
        keep = ~on[self.i]
        self.i, self.j = torch.cat([self.i[keep], i[near]]), torch.cat([self.j[keep], j[near]])
        self.old = torch.where(on, x, self.old)


def _forces(x, pairs, k, a, rrep, ratt):
    i, j = pairs
    e = x[:, i] - x[:, j]
    d = torch.sqrt((e * e).sum(0))
    keep = d < max(rrep, ratt)
    i, e, d = i[keep], e[:, keep], d[keep]
    kk, aa = (v[i] if torch.is_tensor(v) else v for v in (k, a))
    f = torch.where(d < rrep, kk * (rrep - d), -aa * (d - rrep)) / d * e
    return torch.zeros_like(x).index_add_(1, i, f)


def _philox(c, k0, k1):
    """Philox4x32-10 (Salmon et al., SC'11) on four int64 tensors of 32-bit values."""
    M = 0xFFFFFFFF

    def mul(m, v):
        return ((m * (v >> 16) + ((m * (v & 0xFFFF)) >> 16)) >> 16) & M, (m * v) & M

    for _ in range(10):
        h0, l0 = mul(0xD2511F53, c[0])
        h1, l1 = mul(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M
    return c


def _normals(seed, step, agent, community, D, f64):
    """The framework's counter-based normals of one step: (D, n)."""
    z = []
    for sub in range(2 if f64 else 1):
        r = _philox([agent, torch.full_like(agent, step), torch.zeros_like(agent),
                     (community << 8) | sub], seed & 0xFFFFFFFF, seed >> 32)
        if f64:
            u = [((r[2 * k] >> 5).double() * 67108864.0 + (r[2 * k + 1] >> 6).double()) / 2.0 ** 53
                 for k in range(2)]
        else:
            u = [(v >> 8).double() / 2.0 ** 24 for v in r]
        for k in range(0, len(u), 2):
            rad = torch.sqrt(-2 * torch.log(1 - u[k]))
            z += [rad * torch.cos(2 * math.pi * u[k + 1]), rad * torch.sin(2 * math.pi * u[k + 1])]
    return torch.stack(z[:D])


def _stencil(x, lo, dx, m):
    """Nodes and weights of the multilinear stencil around every agent."""
    D = x.shape[0]
    s = [(x[d] - lo[d]) / dx[d] - 0.5 for d in range(D)]
    fl = [torch.floor(v) for v in s]
    for q in range(1 << D):
        node, w = 0, 1.0
        for d in range(D):
            b = (q >> d) & 1
            node = node + torch.clamp(fl[d].long() + b, 0, m - 1) * m ** d
            w = w * ((s[d] - fl[d]) if b else 1 - (s[d] - fl[d]))
        yield node, w


def _exact_agents(case, seed):
    kw, st = _setup(case, seed)
    D, n, steps = kw["dims"], case["n"], case["steps"]
    lo, hi, dt = kw["box_lo"], kw["box_hi"], kw["dt"]
    x = torch.stack([_t(st[k]) for k in "xyz"[:D]])
    agent = torch.arange(n, device=_DEV)
    zero = torch.zeros_like(agent)
    listed_by = case.get("neighbors", "clvd" if case["family"] == "tissue" else "cell")
    grid = _Grid(D, hi[0], kw["skin"] if listed_by == "verlet" else kw["cell_edge"], zero,
                 wide=listed_by in ("verlet", "full"))
    lists = None
    if listed_by in ("clvd", "verlet"):
        lists = _Lists(grid, kw["skin"], kw.get("rebuild_threshold", kw["skin"] / 2), x)
    sq = math.sqrt(np.float32(dt) if case["dtype"] == "f32" else dt)
    if "nodes" in case:
        m = case["nodes"]
        c = _t(st["c"]).reshape((m,) * D)
        g = torch.zeros((D,) + c.shape, dtype=torch.float64, device=_DEV)
        dx = [(hi[d] - lo[d]) / m for d in range(D)]
        mid = (slice(1, -1),) * D

        def shifted(f, d, o):
            return f[tuple(slice(1 + o, m - 1 + o) if k == D - 1 - d else slice(1, -1)
                           for k in range(D))]

    for t in range(steps):
        filed = x
        if kw.get("walls"):
            x = torch.stack([torch.where(x[d] < lo[d], 2 * lo[d] - x[d],
                                         torch.where(x[d] > hi[d], 2 * hi[d] - x[d], x[d]))
                             for d in range(D)])
        pairs = (lists.i, lists.j) if lists else grid.pairs(x, filed)
        dv = _forces(x, pairs, kw["k_rep"], kw["k_att"], kw["r_rep"], kw["r_att"])
        if "nodes" in case:
            sten = list(_stencil(x, lo, dx, m))
            gv = sum(w * g.reshape(D, -1)[:, nd] for nd, w in sten)
            dv = dv + kw["chemotaxis"] * gv / (1 + torch.sqrt((gv * gv).sum(0)))
            u = c.clone().reshape(-1)
            for nd, w in sten:
                amount = kw["secretion"] * dt - kw.get("uptake", 0.0) * dt * c.reshape(-1)[nd]
                u.index_add_(0, nd, w * amount)
            u = u.reshape(c.shape)
            if kw.get("uptake"):
                u = torch.clamp(u, min=0.0)
            g = torch.zeros_like(g)
            for d in range(D):
                g[d][mid] = (shifted(c, d, 1) - shifted(c, d, -1)) / (2 * dx[d])
            lap = sum((shifted(u, d, 1) - 2 * u[mid] + shifted(u, d, -1)) / dx[d] ** 2
                      for d in range(D))
            c = u.clone()
            c[mid] = u[mid] + dt * (kw["diff_D"] * lap - kw["decay"] * u[mid])
        x = x + dv * dt
        if kw.get("sigma"):
            x = x + kw["sigma"] * _normals(seed, t, agent, zero, D, case["dtype"] == "f64") * sq
        if lists:
            lists.check(x)
    out = {k: x[d].cpu() for d, k in enumerate("xyz"[:D])}
    out["N"] = n
    if "nodes" in case:
        out["c"] = c.reshape(-1).cpu()
        out.update({k: g[d].reshape(-1).cpu() for d, k in enumerate(("gx", "gy", "gz")[:D])})
    return out


def _exact_sweep(case, seed):
    descs, states = _sweep_setup(case, seed)
    size = torch.tensor([d["n"] for d in descs], device=_DEV)
    own = torch.repeat_interleave(torch.arange(len(descs), device=_DEV), size)
    first = torch.cumsum(size, 0) - size
    agent = torch.arange(len(own), device=_DEV) - first[own]
    k, a, sig = (_t([d[q] for d in descs])[own] for q in ("k_rep", "k_att", "sigma"))
    x = _t(np.concatenate(states, axis=1))
    lists = _Lists(_Grid(3, [d["L"] for d in descs], 4.0, own), 4.0, 0.5, x)
    for t in range(case["steps"]):
        f = _forces(x, (lists.i, lists.j), k, a, 2.0, 3.0)
        x = x + f * 0.01 + sig * _normals(seed, t, agent, own, 3, False) * math.sqrt(
            np.float32(0.01))
        lists.check(x)
    return {q: x[d].cpu() for d, q in enumerate("xyz")}


def _exact_adjoint(case, seed):
    L, x0, target = _adjoint_setup(case, seed)
    k, a, rho, cut, dt, n = 10.0, 1.0, 2.0, 3.0, 0.01, case["n"]
    x, trace = _t(x0), []
    grid = _Grid(3, L, 3.3, torch.zeros(n, dtype=torch.long, device=_DEV))
    for _ in range(case["steps"]):
        trace.append(x)
        x = x + _forces(x, grid.pairs(x, x), k, a, rho, cut) * dt
    e = x - _t(target)
    loss = float((e * e).sum() / (3 * n))
    lam = 2 * e / (3 * n)
    dth = torch.zeros(3, dtype=torch.float64, device=_DEV)
    for x_t in reversed(trace):
        i, j = grid.pairs(x_t, x_t)
        r = x_t[:, i] - x_t[:, j]
        d = torch.sqrt((r * r).sum(0))
        keep = d < cut
        i, j, r, d = i[keep], j[keep], r[:, keep], d[keep]
        rep = d < rho
        F = torch.where(rep, k * (rho - d), -a * (d - rho))
        dF = torch.where(rep, -k, -a).double()
        lr = (lam[:, i] * r).sum(0) / d
        dth += dt * torch.stack([(lr * torch.where(rep, rho - d, 0.0)).sum(),
                                 (lr * torch.where(rep, 0.0, rho - d)).sum(),
                                 (lr * torch.where(rep, k, a)).sum()])
        dl = lam[:, i] - lam[:, j]
        s, c = F / d, (dF * d - F) / d ** 3
        lam = lam + dt * torch.zeros_like(lam).index_add_(1, i, s * dl + c * r * (r * dl).sum(0))
    return dict(loss=loss, dtheta=dth.cpu(), dx0=list(lam.cpu()), xT=list(x.cpu()))


def _exact_dgadi(case, seed):
    u, src, diff = _dgadi_setup(case, seed)
    D, m = case["dims"], case["nodes"]
    u, src = _t(u), _t(src)
    r = 0.01 / (D * (1.0 / m) ** 2)
    mid = (slice(1, -1),) * D
    T = [torch.zeros(m - 2, m - 2, dtype=torch.float64, device=_DEV) for _ in diff]
    for t, q in zip(T, diff):
        t.diagonal().fill_(1 + 2 * q * r)
        t.diagonal(1).fill_(-q * r)
        t.diagonal(-1).fill_(-q * r)
    inv = [torch.linalg.inv(t) for t in T]
    for _ in range(case["steps"]):
        for f, q in enumerate(diff):
            v = u[f]
            v[mid] += src[mid] * (1.0 - v[mid])
            for axis in reversed(range(D)):  # x is the last dimension
                w = v.movedim(axis, -1)
                inner = (slice(1, -1),) * (D - 1)
                b = w[inner + (slice(1, -1),)].clone()
                b[..., 0] += q * r * w[inner + (0,)]
                b[..., -1] += q * r * w[inner + (m - 1,)]
                w[inner + (slice(1, -1),)] = b @ inv[f]
    return u.cpu()


def _exact_rods(case, seed):
    """The rod colony without growth (rods that divide do so by comparing
    rounded lengths, as agents do)."""
    st = {k: _t(v) for k, v in _rod_state(case, seed).items()}
    half = 1.2 * math.sqrt(case["n"] * 3.8 / math.pi)
    p, dt, n = _ROD, _ROD["dt"], case["n"]
    d, l, m = st["d"], st["l"], st["m"]
    x, y, vx, vy, th, om = (st[k] for k in ("x", "y", "vx", "vy", "theta", "omega"))
    fx, fy, W, pr = (torch.zeros(n, dtype=torch.float64, device=_DEV) for _ in range(4))
    grid = _Grid(2, 2 * half, 4.0, torch.zeros(n, dtype=torch.long, device=_DEV))

    def inside(ax, ay, al, px, py):  # the point clamped to the rod's segment
        q = torch.clamp(torch.hypot(ax - px, ay - py), min=1e-8)
        s = 0.99 * torch.minimum(q, al / 2)
        return s * (px - ax) / q + ax, s * (py - ay) / q + ay

    def online(px, py, ax, ay, ac, as_):  # the point projected on the rod's line
        t = as_ * (ax - px) - ac * (ay - py)
        return t * as_ + px, -t * ac + py

    for _ in range(case["steps"]):
        at = torch.stack([x, y]) + half
        i, j = grid.pairs(at, at)
        c, s = torch.cos(th), torch.sin(th)
        A, B = (x[i], y[i], l[i]), (x[j], y[j], l[j])
        norm = c[i] * s[j] - s[i] * c[j]
        cx, cy = A[0] - B[0], A[1] - B[1]
        cross = norm.abs() > 1e-7
        sc = torch.where(cross, (-s[j] * cx + c[j] * cy) / torch.where(cross, norm, 1.0), 0.0)
        px = torch.where(cross, sc * c[i] + A[0], (A[0] + B[0]) / 2)
        py = torch.where(cross, sc * s[i] + A[1], (A[1] + B[1]) / 2)
        di, dj = torch.hypot(A[0] - px, A[1] - py), torch.hypot(B[0] - px, B[1] - py)
        p1, p2 = inside(*A, px, py), inside(*B, px, py)
        s1 = online(*p2, A[0], A[1], c[i], s[i])
        s2 = online(*p1, B[0], B[1], c[j], s[j])
        in1, in2 = di <= A[2] / 2, dj <= B[2] / 2
        far1 = torch.hypot(A[0] - s1[0], A[1] - s1[1]) > A[2] / 2
        near2 = torch.hypot(B[0] - s2[0], B[1] - s2[1]) < B[2] / 2
        use_s1 = (in1 & ~in2) | (~in1 & ~in2 & ~far1)
        use_s2 = (~in1 & in2) | (~in1 & ~in2 & far1 & near2)
        par = norm.abs() < 1e-6
        q1 = inside(*A, *online(px, py, A[0], A[1], c[i], s[i]))
        q2 = inside(*B, *online(px, py, B[0], B[1], c[j], s[j]))
        xa, ya = (torch.where(par, q1[k], torch.where(use_s1, s1[k], p1[k])) for k in (0, 1))
        xb, yb = (torch.where(par, q2[k], torch.where(use_s2, s2[k], p2[k])) for k in (0, 1))
        rij = torch.hypot(xa - xb, ya - yb)
        hit = (rij > 0) & (rij < (d[i] + d[j]) / 2)
        i, j, xa, ya, xb, yb, rij = (v[hit] for v in (i, j, xa, ya, xb, yb, rij))
        dl, me = d[i] - rij, m[i] / 2
        nx, ny = (xa - xb) / rij, (ya - yb) / rij
        wx, wy = vx[i] - vx[j], vy[i] - vy[j]
        vn = nx * wx + ny * wy
        fn = p["kn"] * dl ** 1.5 - p["gamma_n"] * me * dl * vn
        ft = -torch.minimum(p["gamma_t"] * me * torch.sqrt(dl), p["mu_cc"] * fn)
        gx, gy = fn * nx + ft * (wx - vn * nx), fn * ny + ft * (wy - vn * ny)
        w = (xa - x[i]) * gy - (ya - y[i]) * gx
        aw = W / (m * (d + l) ** 2 / 12 + m * d ** 2) - p["beta_w"] * om
        ax, ay = -p["beta"] * vx + fx / m, -p["beta"] * vy + fy / m
        x, y, th = x + vx * dt, y + vy * dt, th + om * dt
        vx, vy, om = vx + ax * dt, vy + ay * dt, om + aw * dt
        fx, fy, W, pr = (torch.zeros(n, dtype=torch.float64, device=_DEV).index_add_(0, i, v)
                         for v in (gx, gy, w, torch.hypot(gx, gy)))
    st.update(x=x, y=y, vx=vx, vy=vy, theta=th, omega=om, fx=fx, fy=fy, W=W, pressure=pr)
    return {k: None if k == "l_target" else v.cpu() for k, v in st.items()}


def exact(case, seed):
    fam = case["family"]
    if fam == "colony" or case.get("growth"):
        return None  # which agents divide depends on rounded volumes or lengths
    if fam == "chemotaxis":
        return None  # k dt = 2: overlapping pairs overshoot, and roundings grow with every step
    if fam == "sweep":
        n = case["communities"] * (case["n_lo"] + case["n_hi"]) // 2
        return _exact_sweep(case, seed) if n * case["steps"] <= 30_000_000 else None
    if fam == "adjoint":
        return _exact_adjoint(case, seed)
    if fam == "dgadi":
        return _exact_dgadi(case, seed)
    if fam == "rods":
        return _exact_rods(case, seed)
    return _exact_agents(case, seed)
