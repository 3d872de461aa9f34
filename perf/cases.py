"""Timed cases of the cutoff-pair engine: the calls a user's program makes, over the sizes it makes them at.

Every pass is one step of such a program: the new positions are handed over, the cell list is rebuilt and the operator
is mapped over the pairs.  The small cases go through the Python classes with host results; the others through the C ABI
with device buffers, as a simulation that keeps its coordinates on the GPU does.

  python / lists   ParticleSystem.update + pairwise, results as numpy arrays or numbers
  abi              clm_set_positions + clm_run with device pointers
  nl               the same, then the list fetched on the device into buffers of a fixed capacity, and put in the order of
                   its pairs (the library leaves the order, and which end of a pair comes first, open)
  batch            BatchedSystems.update + run, many small independent systems in one step
"""
import ctypes as C
import math

import numpy as np
import torch

import __graft_entry__ as ge

clm = ge.load_package()

LJ_EPS = [[1.0, 1.5], [1.5, 0.5]]
LJ_SIG = [[1.0, 0.8], [0.8, 0.88]]


def _case(name, how, op, dtype, cell, n, rc, rho, layout="uniform", dim=3, prec="exact", n_y=0):
    c = {"how": how, "op": op, "dtype": dtype, "cell": cell, "dim": dim, "n": n, "n_y": n_y, "rc": rc, "rho": rho,
         "layout": layout, "prec": prec}
    return {"name": name, **c} if name else c


def listed():
    return [
        # a small molecule-packing or toy-gas step: a thousand particles, host results, all latency
        _case("soft_forces_1k_py", "python", "soft_forces", "f64", "ortho", 1003, 5.0, 0.1),
        # nearest approach of a small and a larger free cluster (no periodic cell), host results
        _case("mindist_2sets_free_py", "python", "mindist", "f64", "none", 1501, 5.0, 0.1, n_y=4507),
        # an ordinary Lennard-Jones MD step, 32,000 particles in a cubic box
        _case("lj_f32_cubic_32k", "abi", "lj_forces", "f32", "ortho", 32000, 2.5, 0.8, layout="fcc"),
        # the largest Lennard-Jones step: a million particles in a sheared cell
        _case("lj_f32_triclinic_1m", "abi", "lj_forces", "f32", "tri", 1048576, 2.5, 0.8, layout="fcc"),
        # the same system in Float64, a quarter of the size
        _case("lj_f64_triclinic_256k", "abi", "lj_forces", "f64", "tri", 256000, 2.5, 0.8, layout="fcc"),
        # long-cutoff soft repulsion in Float64 with FP32 pair arithmetic (about 107 partners per particle and side)
        _case("soft_forces_f64_split_100k", "abi", "soft_forces", "f64", "ortho", 100000, 8.0, 0.1, prec="split"),
        # the neighbour list of the library's documentation size: 100,000 points, cutoff 8, 1.1e7 pairs
        _case("nl_f64_100k", "nl", "nl", "f64", "ortho", 100000, 8.0, 0.1),
        # a two-dimensional neighbour list of an odd size in Float32
        _case("nl_f32_2d_200k", "nl", "nl", "f32", "ortho", 200003, 3.0, 0.5, dim=2),
        # gradient of a two-type mixture's energy with respect to positions, cell and pair parameters
        _case("adjoint_f32_200k", "abi", "lj_adjoint", "f32", "ortho", 200000, 2.5, 1.2, layout="mix"),
        # mean pairwise radial velocities of two catalogues in 50 logarithmic bins
        _case("rhist_2sets_f64_100k", "abi", "rhist", "f64", "ortho", 100003, 25.0, 0.128, n_y=100003),
        # the same in two dimensions
        _case("rhist_2sets_2d_f64_100k", "abi", "rhist", "f64", "ortho", 100003, 25.0, 0.128, dim=2, n_y=100003),
        # a thousand independent small systems in one step: neighbour lists and energies
        {"name": "batch_nl_energy_f64_1k", "how": "batch", "op": "nl+soft_energy", "dtype": "f64", "cell": "ortho",
         "dim": 3, "nsys": 1024, "nmin": 200, "nmax": 2000, "rc": 6.0, "rho": 0.1, "prec": "exact", "graph": True},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["python", "mindist", "lj32", "lj32", "lj64", "soft", "nl", "nl2d", "adjoint", "rhist", "rhist2d", "batch"])
    cell = rng.choice(["ortho", "tri"])
    if kind == "python" and rng.random() < 0.5:
        return _case(None, "python", "lj_forces", rng.choice(["f32", "f64"]), cell, 4 * rng.randint(5, 17) ** 3,
                     rng.uniform(2.2, 3.0), rng.uniform(0.6, 1.0), layout="fcc")
    if kind == "python":
        return _case(None, "python", "soft_forces", rng.choice(["f32", "f64"]), cell, _logint(rng, 500, 20000),
                     rng.uniform(2.5, 3.5), rng.uniform(0.1, 0.4))
    if kind == "mindist":
        n = _logint(rng, 500, 50000)
        return _case(None, "python", "mindist", rng.choice(["f32", "f64"]), rng.choice(["none", "ortho"]), n, 5.0, 0.1,
                     n_y=_logint(rng, n, 4 * n))
    if kind in ("lj32", "lj64"):
        m = rng.randint(8, 63 if kind == "lj32" else 40)
        return _case(None, "abi", "lj_forces", "f32" if kind == "lj32" else "f64", cell, 4 * m ** 3, rng.uniform(2.2, 3.0),
                     rng.uniform(0.6, 1.0), layout="fcc")
    if kind == "soft":
        return _case(None, "abi", rng.choice(["soft_forces", "soft_energy"]), "f64", cell, _logint(rng, 4000, 120000),
                     rng.uniform(5.0, 8.0), 0.1, prec=rng.choice(["exact", "split"]))
    if kind == "nl":
        return _case(None, "nl", "nl", rng.choice(["f32", "f64"]), rng.choice(["ortho", "tri", "none"]),
                     _logint(rng, 4000, 100000), rng.uniform(4.0, 8.0), 0.1)
    if kind == "nl2d":
        return _case(None, "nl", "nl", rng.choice(["f32", "f64"]), cell, _logint(rng, 4000, 250000), rng.uniform(2.0, 4.0), 0.5,
                     dim=2)
    if kind == "adjoint":
        return _case(None, "abi", "lj_adjoint", "f32", "ortho", _logint(rng, 10000, 200000), rng.uniform(2.2, 2.6), 1.2,
                     layout="mix")
    if kind in ("rhist", "rhist2d"):
        n = _logint(rng, 10000, 100000)
        return _case(None, "abi", "rhist", "f64", cell, n, rng.uniform(12.0, 20.0) if kind == "rhist" else 25.0, 0.128,
                     dim=3 if kind == "rhist" else 2, n_y=_logint(rng, 10000, 100000))
    return {"how": "batch", "op": "nl+soft_energy", "dtype": rng.choice(["f32", "f64"]), "cell": "ortho", "dim": 3,
            "nsys": _logint(rng, 64, 1024), "nmin": 200, "nmax": rng.randint(400, 2000), "rc": rng.uniform(5.0, 6.0),
            "rho": 0.1, "prec": rng.choice(["exact", "split"]), "graph": rng.random() < 0.5}


# ------------------------------------------------------------------------------------------------ inputs
def _dt(case):
    return torch.float64 if case["dtype"] == "f64" else torch.float32


def _cell(case):
    """Cell matrix (columns are the cell vectors) of volume n / rho; without a periodic cell, the sides of the cluster."""
    d = case["dim"]
    side = (max(case["n"], case["n_y"]) / case["rho"]) ** (1.0 / d)
    M = np.eye(d) * side
    if case["cell"] == "tri":
        M[0, 1] = 0.2 * side
        if d == 3:
            M[0, 2], M[1, 2] = 0.1 * side, 0.15 * side
    return M


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * (seed + 1))
    return g


def _positions(case, g, M, n):
    """Uniform points; a jittered fcc crystal; or a jittered fcc crystal with vacancies at random sites (mixtures)."""
    d = case["dim"]
    if case["layout"] == "uniform":
        f = torch.rand((n, d), generator=g, device="cuda", dtype=torch.float64)
        return (f @ torch.from_numpy(M.T.copy()).cuda()).to(_dt(case))
    m = math.ceil(round((n / 4) ** (1.0 / 3.0), 6))
    a = torch.arange(m, device="cuda", dtype=torch.float64)
    grid = torch.stack(torch.meshgrid(a, a, a, indexing="ij"), -1).reshape(-1, 1, 3)
    basis = torch.tensor([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]], device="cuda", dtype=torch.float64)
    f = ((grid + basis) / m).reshape(-1, 3)
    if f.shape[0] > n or case["layout"] == "mix":
        f = f[torch.randperm(f.shape[0], generator=g, device="cuda")[:n]]
    x = f @ torch.from_numpy(M.T.copy()).cuda()
    return (x + 0.05 * torch.randn(x.shape, generator=g, device="cuda", dtype=torch.float64)).to(_dt(case)).contiguous()


def _inputs(case, seed):
    g = _generator(seed)
    if case["how"] == "batch":
        # log-uniform sizes in a mixed order, the same for every seed
        share = (np.random.default_rng(1).permutation(case["nsys"]) + 0.5) / case["nsys"]
        sizes = (case["nmin"] * (case["nmax"] / case["nmin"]) ** share).astype(np.int64)
        off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
        side = (sizes / case["rho"]) ** (1.0 / 3.0)
        f = torch.rand((int(off[-1]), 3), generator=g, device="cuda", dtype=torch.float64)
        per = torch.repeat_interleave(torch.from_numpy(side).cuda(), torch.from_numpy(sizes).cuda())
        return {"x": (f * per[:, None]).to(_dt(case)), "off": off, "side": side}
    M = _cell(case)
    inp = {"M": M, "x": _positions(case, g, M, case["n"])}
    if case["n_y"]:
        inp["y"] = _positions(case, g, M, case["n_y"])
    if case["layout"] == "mix":
        inp["types"] = (torch.rand(case["n"], generator=g, device="cuda") >= 0.8).to(torch.int32)
    if case["op"] == "rhist":
        for s in ("x", "y"):
            inp["v" + s] = 300.0 * torch.randn(inp[s].shape, generator=g, device="cuda", dtype=_dt(case))
        inp["bins"] = 10.0 ** np.linspace(math.log10(0.1), math.log10(case["rc"]), 51)
    return inp


def _operator(case):
    return {"soft_forces": clm.SoftForces, "lj_forces": clm.LennardJonesForces, "mindist": clm.MinimumDistance}[case["op"]]()


class _Handle:
    """A library handle driven through the C ABI, with the operator's parameter and output blocks."""

    def __init__(self, case, inp):
        self.abi = clm._abi
        self.L = self.abi.load()
        self.h = C.c_void_p()
        self.inp, self.case = inp, case
        f64 = case["dtype"] == "f64"
        self.ok(self.L.clm_create(self.abi.CLM_F64 if f64 else self.abi.CLM_F32, case["dim"], 2 if case["n_y"] else 1, C.byref(self.h)))
        kind = {"ortho": self.abi.CLM_ORTHO, "tri": self.abi.CLM_TRICLINIC, "none": self.abi.CLM_NONPERIODIC}[case["cell"]]
        M = np.ascontiguousarray(inp["M"].flatten(order="F"))
        self.ok(self.L.clm_set_box(self.h, M.ctypes.data_as(C.POINTER(C.c_double)), kind, case["rc"], 1))
        self.ok(self.L.clm_set_precision(self.h, self.abi.CLM_PREC_SPLIT if case["prec"] == "split" else self.abi.CLM_PREC_EXACT))
        self.p, self.o = self.abi.OpParams(), self.abi.Outputs()
        if case["op"].startswith("lj"):
            self.p.p[0], self.p.p[1], self.p.p[2], self.p.p[3] = 1.0, 1.0, 4.0, 4.0
        self.p.params_on_device = 1
        self.o.out_on_device = 1
        if "types" in inp:
            self.eps = torch.tensor(LJ_EPS, dtype=torch.float64, device="cuda")
            self.sig = torch.tensor(LJ_SIG, dtype=torch.float64, device="cuda")
            self.p.ntypes, self.p.types_x = 2, inp["types"].data_ptr()
            self.p.eps_table, self.p.sig_table = self.eps.data_ptr(), self.sig.data_ptr()
        if case["op"] in ("lj_forces", "soft_forces", "lj_adjoint"):
            self.forces = torch.empty_like(inp["x"])
            self.o.forces_x = self.forces.data_ptr()
        if case["op"] == "lj_adjoint":
            self.adj = np.zeros(15)
            self.o.adjoint = self.adj.ctypes.data
        if case["op"] == "rhist":
            self.bins = torch.from_numpy(inp["bins"]).cuda()
            self.hc = torch.empty(50, dtype=torch.int64, device="cuda")
            self.hs = torch.empty(50, dtype=torch.float64, device="cuda")
            self.p.nbins, self.p.bins = 50, self.bins.data_ptr()
            self.p.vel_x, self.p.vel_y = inp["vx"].data_ptr(), inp["vy"].data_ptr()
            self.o.hist_count, self.o.hist_sum = self.hc.data_ptr(), self.hs.data_ptr()

    def ok(self, status):
        if status:
            buf = C.create_string_buffer(512)
            self.L.clm_last_error(self.h, buf, 512)
            raise RuntimeError("clm status %d: %s" % (status, buf.value.decode()))

    def step(self):
        self.ok(self.L.clm_set_positions(self.h, 0, self.inp["x"].data_ptr(), self.case["n"], 1))
        if self.case["n_y"]:
            self.ok(self.L.clm_set_positions(self.h, 1, self.inp["y"].data_ptr(), self.case["n_y"], 1))
        self.ok(self.L.clm_run(self.h, self.abi.OP[self.case["op"]], C.byref(self.p), C.byref(self.o)))

    def __del__(self):
        if self.h:
            self.L.clm_destroy(self.h)
            self.h = None


class _ListBuffers:
    """Device buffers of a program that keeps its neighbour list in a fixed capacity, a little above the expected pairs,
    sorted by the lower particle of a pair and then the other (both of one system, so that it is less than `span` away)."""

    def __init__(self, case, n):
        self.cap = int(1.05 * _pairs(case)) + 8192
        self.span = case["nmax"] if case["how"] == "batch" else n
        self.end = n * self.span
        narrow = self.end < 2 ** 31
        self.i, self.j = (torch.empty(self.cap, dtype=torch.int64, device="cuda") for _ in range(2))
        self.key = torch.empty(self.cap, dtype=torch.int32 if narrow else torch.int64, device="cuda")
        self.d = torch.empty(self.cap, dtype=_dt(case), device="cuda")

    def fill(self, L, h, count):
        """The list in the order of its pairs as lower * span + (upper - lower), and 0 for the rest of the distances."""
        status = L.clm_nl_fetch(h, self.i.data_ptr(), self.j.data_ptr(), self.d.data_ptr(), self.cap, 0, 1)
        if status:
            raise RuntimeError("clm status %d" % status)
        i, j = self.i[:count], self.j[:count]
        self.key[:count] = torch.add((i - j).abs_(), torch.minimum(i, j), alpha=self.span)
        self.key[count:] = self.end
        self.d[count:] = 0
        key, at = torch.sort(self.key)
        return {"pair": key, "d": self.d[at], "count": count}


def prepare(case, seed):
    """Positions (and velocities or types) on the GPU, and the system object or handle a program keeps between steps."""
    inp = _inputs(case, seed)
    state = {"case": case, "inp": inp}
    if case["how"] == "batch":
        state["sys"] = clm.BatchedSystems(positions=inp["x"], offsets=inp["off"], unitcells=np.repeat(inp["side"][:, None], 3, axis=1),
                                          cutoff=case["rc"], dtype=np.float64 if case["dtype"] == "f64" else np.float32,
                                          precision=case["prec"], graph=case["graph"])
        state["ops"] = (clm.NeighborList(), clm.SoftEnergy())
        state["list"] = _ListBuffers(case, int(inp["off"][-1]))
    elif case["how"] == "python":
        cell = None if case["cell"] == "none" else (inp["M"] if case["cell"] == "tri" else np.diag(inp["M"]).copy())
        state["sys"] = clm.ParticleSystem(xpositions=inp["x"], ypositions=inp.get("y"), unitcell=cell, cutoff=case["rc"],
                                          dtype=np.float64 if case["dtype"] == "f64" else np.float32, precision=case["prec"])
        state["op"] = _operator(case)
    else:
        state["handle"] = _Handle(case, inp)
        if case["how"] == "nl":
            state["list"] = _ListBuffers(case, case["n"])
    return state


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    case, inp = state["case"], state["inp"]
    if case["how"] == "batch":
        sys = state["sys"]
        sys.update(positions=inp["x"])
        lists, energy = sys.run(*state["ops"])
        h = sys._handle
        return {"counts": lists.counts, "energy": energy, "list": state["list"].fill(h.L, h.h, lists.total)}
    if case["how"] == "python":
        sys = state["sys"]
        sys.update(xpositions=inp["x"], ypositions=inp.get("y"))
        r = clm.pairwise(state["op"], sys)
        return {"energy": r.energy, "forces": r.forces} if case["op"] != "mindist" else {"i": r[0], "j": r[1], "d": r[2]}
    h = state["handle"]
    h.step()
    if case["how"] == "nl":
        return state["list"].fill(h.L, h.h, h.o.count)
    if case["op"] == "rhist":
        return {"counts": h.hc, "sums": h.hs}
    out = {"energy": h.o.scalar}
    if case["op"] != "soft_energy":
        out["forces"] = h.forces
    if case["op"] == "lj_adjoint":
        out["virial"], out["dU_deps"], out["dU_dsigma"] = h.adj[:9], h.adj[9:12], h.adj[12:15]
    return out


# ------------------------------------------------------------------------------------------------ what a pass needs
_FLOPS = {"soft_forces": 15.0, "soft_energy": 4.0, "lj_forces": 20.0, "mindist": 1.0, "nl": 1.0, "lj_adjoint": 42.0, "rhist": 11.0,
          "nl+soft_energy": 5.0}


def _ball(case):
    return math.pi * case["rc"] ** 2 if case["dim"] == 2 else 4.0 / 3.0 * math.pi * case["rc"] ** 3


def _pairs(case):
    """Pairs within the cutoff expected at uniform density."""
    ball = _ball(case)
    if case["how"] == "batch":
        lo, hi = case["nmin"], case["nmax"]
        return case["nsys"] * (hi - lo) / math.log(hi / lo) * case["rho"] * ball / 2
    n, m = case["n"], case["n_y"]
    return (n * m / max(n, m) if m else n / 2) * case["rho"] * ball


def work(case):
    """Inputs read and outputs written once; eight operations for a pair's distance and the operator's own."""
    d, w, pairs = case["dim"], 8 if case["dtype"] == "f64" else 4, _pairs(case)
    n = pairs / (case["rho"] * _ball(case) / 2) if case["how"] == "batch" else case["n"] + case["n_y"]
    b = n * d * w
    if case["op"] in ("lj_forces", "soft_forces", "lj_adjoint", "rhist"):
        b += n * d * w
    if "nl" in case["op"].split("+"):
        b += pairs * (16 + w)
    return {"bytes": b, "flops": pairs * (8 + _FLOPS[case["op"]])}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
class _Grid:
    """Points binned into cells at least a cutoff wide, as padded rows of point numbers (-1: none)."""

    def __init__(self, x, M, lo, nc, periodic):
        Minv = torch.linalg.inv(M)
        f = (x - lo) @ Minv.T
        if periodic:
            f = f - torch.floor(f)
        self.x = lo + f @ M.T
        c = (f * nc).long().clamp(min=0)
        c = torch.minimum(c, nc - 1)
        li = torch.zeros(x.shape[0], dtype=torch.long, device=x.device)
        for a in range(x.shape[1]):
            li = li * nc[a] + c[:, a]
        total = int(nc.prod())
        cnt = torch.bincount(li, minlength=total)
        order = torch.argsort(li, stable=True)
        start = torch.cumsum(cnt, 0) - cnt
        rank = torch.arange(x.shape[0], device=x.device) - start[li[order]]
        self.rows = torch.full((total, int(cnt.max())), -1, dtype=torch.long, device=x.device)
        self.rows[li[order], rank] = order


def _pairs64(x, y, M, rc, periodic):
    """Every (i, j, dx) with |dx| <= rc, dx = x_i - (nearest image of y_j), in blocks; x and y the same tensor: each pair twice."""
    d = x.shape[1]
    if not periodic:
        both = torch.cat([x, y])
        lo = both.min(0).values - rc
        M = torch.diag(both.max(0).values + rc - lo)
    else:
        lo = torch.zeros(d, dtype=x.dtype, device=x.device)
    height = 1.0 / torch.linalg.inv(M).norm(dim=1)
    nc = torch.clamp((height / rc * (1 - 1e-9)).long(), min=1, max=4096)
    gx = _Grid(x, M, lo, nc, periodic)
    gy = gx if y is x else _Grid(y, M, lo, nc, periodic)
    cells = torch.cartesian_prod(*[torch.arange(int(v), device=x.device) for v in nc])
    block = max(1, 20_000_000 // max(1, gx.rows.shape[1] * gy.rows.shape[1]))
    for shift in torch.cartesian_prod(*[torch.arange(-1, 2, device=x.device)] * d):
        to = cells + shift
        turn = torch.div(to, nc, rounding_mode="floor")
        inside = torch.ones(cells.shape[0], dtype=torch.bool, device=x.device) if periodic else (turn == 0).all(1)
        to = to - turn * nc
        lj = torch.zeros(cells.shape[0], dtype=torch.long, device=x.device)
        for a in range(d):
            lj = lj * nc[a] + to[:, a]
        move = turn.to(x.dtype) @ M.T
        for b in range(0, cells.shape[0], block):
            e = slice(b, b + block)
            ri, rj = gx.rows[e][:, :, None], gy.rows[lj[e]][:, None, :]
            keep = (ri >= 0) & (rj >= 0) & inside[e][:, None, None]
            dx = gx.x[ri.clamp(min=0)] - (gy.x[rj.clamp(min=0)] + move[e][:, None, None, :])
            d2 = dx.square().sum(-1)
            keep &= d2 <= rc * rc
            if y is x:
                keep &= ri != rj
            at = keep.nonzero(as_tuple=True)
            yield ri.expand_as(keep)[at], rj.expand_as(keep)[at], dx[at], d2[at]


def _list64(case, keys, dist):
    d = torch.cat(dist)[torch.argsort(torch.cat(keys))]
    return {"pair": None, "d": torch.nn.functional.pad(d, (0, int(1.05 * _pairs(case)) + 8192 - d.numel())), "count": None}


def _batch64(case, inp):
    off, energy, keys, dist = inp["off"], [], [], []
    x, rc = inp["x"].double(), case["rc"]
    n = int(off[-1])
    for s in range(case["nsys"]):
        p, L = x[off[s]:off[s + 1]], float(inp["side"][s])
        dx = p[:, None, :] - p[None, :, :]
        dx = dx - L * torch.round(dx / L)
        d2 = dx.square().sum(-1)
        i, j = torch.triu(d2 <= rc * rc, diagonal=1).nonzero(as_tuple=True)
        r = d2[i, j].sqrt()
        energy.append((rc - r).square().sum())
        keys.append((i + int(off[s])) * n + (j + int(off[s])))
        dist.append(r)
    if case["dtype"] == "f32":  # as in exact()
        return {"counts": None, "energy": torch.stack(energy), "list": {"pair": None, "d": None, "count": None}}
    return {"counts": None, "energy": torch.stack(energy), "list": _list64(case, keys, dist)}


def exact(case, seed):
    inp = _inputs(case, seed)
    if case["how"] == "batch":
        return _batch64(case, inp)
    x = inp["x"].double()
    y = inp["y"].double() if "y" in inp else x
    M = torch.from_numpy(inp["M"]).cuda()
    blocks = _pairs64(x, y, M, case["rc"], case["cell"] != "none")
    op, d, rc = case["op"], case["dim"], case["rc"]
    if op == "nl" and case["dtype"] == "f32":
        return None  # Float32 distances put some pairs at the cutoff on its other side: the list is another one
    if op == "nl":
        keys, dist = [], []
        for i, j, _, d2 in blocks:
            once = i < j
            keys.append((i * case["n"] + j)[once])
            dist.append(d2[once].sqrt())
        return _list64(case, keys, dist)
    if op == "mindist":
        best = min((float(b[3].min()) for b in blocks if b[3].numel()), default=math.inf)
        return {"i": None, "j": None, "d": math.sqrt(best)}
    if op == "rhist":
        edges = torch.from_numpy(inp["bins"]).cuda()
        sums = torch.zeros(52, dtype=torch.float64, device="cuda")
        vx, vy = inp["vx"].double(), inp["vy"].double()
        for i, j, dx, d2 in blocks:
            r = d2.sqrt()
            term = ((vx[i] - vy[j]) * dx).sum(-1) / r
            at = torch.bucketize(r, edges)
            sums += torch.bincount(at, weights=term, minlength=52)
        return {"counts": None, "sums": sums[1:51]}
    typed = "types" in inp
    if typed:
        t = inp["types"].long()
        eps_t, sig_t = (torch.tensor(v, dtype=torch.float64, device="cuda") for v in (LJ_EPS, LJ_SIG))
    energy = torch.zeros((), dtype=torch.float64, device="cuda")
    force, virial = torch.zeros_like(x), torch.zeros((3, 3), dtype=torch.float64, device="cuda")
    de, ds = (torch.zeros(3, dtype=torch.float64, device="cuda") for _ in range(2))
    for i, j, dx, d2 in blocks:  # each pair twice: the sums over pairs are halved
        if op.startswith("soft"):
            r = d2.sqrt()
            u, g = (rc - r).square(), -2.0 * (rc - r) / r
        else:
            eps, sig = (eps_t[t[i], t[j]], sig_t[t[i], t[j]]) if typed else (1.0, 1.0)
            s6 = (sig * sig / d2) ** 3
            u, g = eps * 4.0 * (s6 * s6 - s6), eps * (-48.0 * s6 * s6 + 24.0 * s6) / d2
        energy += 0.5 * u.sum()
        force.index_add_(0, i, -g[:, None] * dx)
        if typed:
            virial += 0.5 * (dx * g[:, None]).T @ dx
            cls = t[i] + t[j]
            de.index_add_(0, cls, 0.5 * u / eps)
            ds.index_add_(0, cls, 0.5 * eps * (48.0 * s6 * s6 - 24.0 * s6) / sig)
    out = {"energy": float(energy)}
    if op != "soft_energy":
        out["forces"] = force
    if typed:
        out["virial"], out["dU_deps"], out["dU_dsigma"] = virial.reshape(-1), de, ds
    return out
