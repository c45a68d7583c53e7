"""Workloads that a user of soil_b200 runs, for timing and for checking results.

A case is a dict of plain values.  Its `kind` says how the framework is used:

  run      one resident system that a program keeps and advances: a pass is
           `System.step(K)`, after which the program reads the state and the
           lists where they are, on the GPU (`System.view`)
  job      one simulation from start to end: host arrays in, set up, K steps,
           final state and neighbor list back on the host, system closed
  batch    many independent boxes kept in one `Batch`: K batched steps, then
           every box's positions and velocities read into pinned host memory
  serve    jobs submitted to a `Server` all at once; a pass ends with the last
           job's result
  binsort  the spatial sort's permutation of positions a program holds on the
           GPU (`soil_bin_sort_noalloc`)

The particles are those of soil_b200.workloads: spheres thrown at random into
a cubic box at volume fraction `phi`, unit-normal velocities, mass 1.  `mono`
spheres have diameter 1; otherwise radii are uniform in [0.4, 0.6].
"""
import ctypes
import math

import numpy as np
import torch

from soil_b200 import abi, system, workloads

RMIN, RMAX, SKIN = 0.4, 0.6, 0.1
MEAN_R3 = (RMAX ** 4 - RMIN ** 4) / (4.0 * (RMAX - RMIN))


def listed():
    return [
        # The smallest systems users step one at a time: launches, barriers
        # and host decisions are everything.
        _run("tiny-1000", 1000, 0.45, steps=200),
        # The plain 32,768-sphere box without a consumer (free flight, mono).
        _run("plain-32768", 32768, 0.30, steps=200, k=0.0, mono=True, dt=1e-3),
        # A served-size box near its upper end, with the FP32 prefilter those jobs use.
        _run("dense-200003-fp32", 200003, 0.50, steps=50, fp32=True),
        # The large headline box: a dense packing with mixed radii.
        _run("dense-4194304", 4194304, 0.50, steps=16),
        # A small box under Lees-Edwards shear: every step rebuilds its lists.
        _run("shear-8009", 8009, 0.35, steps=40, rate=0.15),
        # The large sheared box of equal spheres.
        _run("shear-1048576", 1048576, 0.40, steps=8, rate=0.1, mono=True),
        # Parameter study of small boxes, half of them sheared.
        _batch("batch-64-small", 64, 256, 4096, steps=30),
        # The batched configuration's whole range of sizes.
        _batch("batch-128", 128, 256, 65536, steps=30),
        # A burst of jobs at a server.
        dict(name="serve-10", kind="serve", jobs=10, nmin=1024, nmax=32768, steps=150),
        # One simulation from host arrays to host results.
        _job("job-65537", 65537, 0.45, steps=40),
        # A slab compressed along x with a shrink-wrapped z, full lists
        # (newton off), driven phase by phase by the host's own schedule.
        _job("job-slab-30011", 30011, 0.40, steps=20, newton=False, squeeze=-0.5, slab=True,
             phases=True),
        # The spatial sort alone, near the largest grid it serves.
        dict(name="binsort-2000003", kind="binsort", n=2000003, phi=0.50),
    ]


def _run(name, n, phi, steps, **kw):
    c = dict(name=name, kind="run", n=n, phi=phi, steps=steps, k=1e3, mono=False, dt=1e-4,
             rate=0.0, fp32=False, newton=True)
    c.update(kw)
    return c


def _job(name, n, phi, steps, **kw):
    c = dict(_run(name, n, phi, steps), kind="job", squeeze=0.0, slab=False, phases=False)
    c.update(kw)
    return c


def _batch(name, boxes, nmin, nmax, steps):
    return dict(name=name, kind="batch", boxes=boxes, nmin=nmin, nmax=nmax, steps=steps)


def draw(rng):
    def logn(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["run"] * 5 + ["job"] * 2 + ["batch"] * 2 + ["serve", "binsort"])
    phi = round(rng.uniform(0.20, 0.55), 3)
    if kind == "run":
        mono = rng.random() < 0.4
        k = 0.0 if mono and rng.random() < 0.5 else 1e3
        rate = round(rng.uniform(0.01, 0.2), 3) if k and rng.random() < 0.4 else 0.0
        n = logn(1000, 2000000)
        steps = max(4, min(200, int(4e6 / n)))
        if rate:
            steps = max(3, steps // 4)
        c = _run("", n, phi, steps, k=k, mono=mono, dt=1e-4 if k else 1e-3, rate=rate,
                 fp32=rng.random() < 0.4, newton=rng.random() < 0.8)
    elif kind == "job":
        slab = rng.random() < 0.4
        c = _job("", logn(1024, 262144), phi, rng.randint(10, 40), mono=rng.random() < 0.4,
                 fp32=rng.random() < 0.4, newton=rng.random() < 0.7, slab=slab,
                 squeeze=round(rng.uniform(-0.8, 0.8), 2) or 0.1 if slab or rng.random() < 0.4
                 else 0.0,
                 phases=slab and rng.random() < 0.5)
    elif kind == "batch":
        boxes, nmax = logn(16, 128), logn(1024, 65536)
        c = _batch("", boxes, 256, nmax, max(5, min(40, int(1e8 / (boxes * nmax)))))
    elif kind == "serve":
        c = dict(kind="serve", jobs=rng.randint(2, 14), nmin=1024, nmax=logn(4096, 32768),
                 steps=rng.randint(80, 200))
    else:
        c = dict(kind="binsort", n=logn(10000, 2000000), phi=round(rng.uniform(0.3, 0.5), 3))
    c.pop("name", None)
    return c


# ---- inputs ------------------------------------------------------------------


def _generator(seed, stream=0):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + stream * 7919 + 17) % (1 << 62))
    return g


def _side(c):
    """Box edge: n spheres of the case's mean volume at its volume fraction."""
    r3 = 0.125 if c["mono"] else MEAN_R3
    return (c["n"] * 4.0 / 3.0 * math.pi * r3 / c["phi"]) ** (1.0 / 3.0)


def _particles(c, seed, stream=0):
    """(positions, velocities, radii) of a case, on the GPU."""
    g, n = _generator(seed, stream), c["n"]
    kw = dict(generator=g, device="cuda", dtype=torch.float64)
    x = torch.rand((n, 3), **kw) * _side(c)
    v = torch.randn((n, 3), **kw)
    v -= v.mean(dim=0)
    r = torch.full((n,), 0.5, dtype=torch.float64, device="cuda") if c["mono"] else \
        RMIN + (RMAX - RMIN) * torch.rand((n,), **kw)
    return x, v, r


def _workload(c, seed, stream=0):
    x, v, r = (t.cpu().numpy() for t in _particles(c, seed, stream))
    kw = dict(filter=abi.SOIL_FILTER_FP32_RECHECK if c["fp32"] else abi.SOIL_FILTER_FP64,
              newton=1 if c["newton"] else 0)
    if c["mono"]:  # relative skin on the diameter
        cut, cfg = r, workloads.default_cfg(skin_fraction=1.0 + SKIN, **kw)
    else:          # additive skin on the sum of the radii
        cut, cfg = r + 0.5 * SKIN, workloads.default_cfg(additive_skin=SKIN, **kw)
    return workloads.Workload(c["kind"], c["n"], _side(c), x, v, r, cut, cfg, c["dt"], c["steps"],
                              harmonic_k=c["k"], shear_rate=c["rate"], seed=seed)


def _boxes(c):
    """The boxes of a batch or the jobs of a burst: sizes log-uniform in
    [nmin, nmax], every other one sheared."""
    rs = np.random.RandomState(c["nmax"] + c["steps"])
    out = []
    for i in range(c.get("boxes") or c["jobs"]):
        n = int(round(math.exp(rs.uniform(math.log(c["nmin"]), math.log(c["nmax"])))))
        phi = rs.uniform(0.20, 0.55)
        rate = 0.01 + 0.19 * rs.random_sample()
        out.append(_run("", n, phi, c["steps"] + (i * 7) % 31 if c["kind"] == "serve" else c["steps"],
                        rate=rate if i % 2 else 0.0, fp32=c["kind"] == "serve"))
    return out


def _room(c):
    """Entries of the array that a program keeps its own copy of the list in."""
    return int(c["n"] * _pairs_per_atom(c)[0] * (2 if c["newton"] else 4)) + 4096


def _grid(L, cut):
    """Bin grid of a cubic box of edge L with two ghost layers a side."""
    ni = max(1, int(L / cut))
    return ni + 4, L / ni, -2.0 * (L / ni)


_shared = {}


def _context():
    if "ctx" not in _shared:
        _shared["ctx"] = system.Context(0)
    return _shared["ctx"]


# ---- passes ------------------------------------------------------------------


class _Server:
    """A server with the context that its loop thread owns."""

    def __init__(self):
        from soil_b200.serve import Server
        self.ctx = system.Context(0)
        self.server = Server(self.ctx)

    def __del__(self):
        self.server.close()


def prepare(case, seed):
    c = case
    if c["kind"] == "run":
        return dict(case=c, sys=system.from_workload(_context(), _workload(c, seed)),
                    list=torch.empty(_room(c), dtype=torch.int32, device="cuda"))
    if c["kind"] == "job":
        return dict(case=c, ctx=_context(), w=_workload(c, seed),
                    list=np.zeros(_room(c), np.uint32))
    if c["kind"] == "batch":
        ctx = _context()
        members = [system.from_workload(ctx, _workload(b, seed, i))
                   for i, b in enumerate(_boxes(c))]
        batch = system.Batch(ctx)
        for s in members:
            batch.add(s)
        ns = [s.counts().nlocal for s in members]
        host = torch.empty((2, sum(ns), 3), dtype=torch.float64, pin_memory=True)
        ends = np.cumsum([0] + ns)
        return dict(case=c, batch=batch, members=members, ends=ends, host=host, np=host.numpy())
    if c["kind"] == "serve":
        return dict(case=c, srv=_Server(),
                    jobs=[_workload(b, seed, i) for i, b in enumerate(_boxes(c))])
    L = _side(dict(c, mono=False))
    x = torch.rand((3, c["n"]), generator=_generator(seed), device="cuda", dtype=torch.float64) * L
    nb, size, origin = _grid(L, 2 * RMAX + SKIN)
    f3, i3 = ctypes.c_double * 3, ctypes.c_int32 * 3
    out = torch.empty((2, c["n"]), dtype=torch.int32, device="cuda")
    return dict(case=c, ctx=_context(), x=x, out=out,
                grid=(f3(*[origin] * 3), f3(*[size] * 3), i3(*[nb] * 3), f3(0.0, 0.0, 0.0),
                      f3(L, L, L), f3(0.0, 0.0, 0.0)))


class _OnDevice:
    """A device array of a system, as torch reads it; keeps the system alive."""

    def __init__(self, owner, ptr, n, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=(n,), typestr=typestr, data=(ptr, False),
                                             version=3, strides=None)


def _view(s, room):
    """The locals' state of a system where it is, and its neighbor list copied
    to the program's own array (entries past its end are -1)."""
    v = s.view()
    n = v.nlocal

    def at(ptr, m, t):
        if not m:
            return torch.empty(0, dtype=torch.float64 if t == "<f8" else torch.int32, device="cuda")
        return torch.as_tensor(_OnDevice(s, ptr, m, t), device="cuda")

    out = {k: at(getattr(v, k), n, "<f8")
           for k in ("x", "y", "z", "vx", "vy", "vz", "fx", "fy", "fz")}
    out["tag"] = at(v.tag, n, "<i4")
    out["offsets"] = at(v.neighbor_offsets, n + 1, "<i4")
    room[:v.npairs].copy_(at(v.neighbor_indices, v.npairs, "<i4"))
    room[v.npairs:].fill_(-1)
    out["indices"] = room
    return out


PHASES = ("deform", "initial", "decide_rebuild", "remove_ghosts", "zero_forces", "shrink_wrap",
          "pbc", "sort", "borders", "forward_comm", "neighbor", "force", "reverse_comm", "final")


def _run_job(ctx, c, w, room):
    s = system.System(ctx, w.box, w.cfg, w.dt)
    rc = s.register_column("radius", 1, abi.SOIL_COL_FORWARD)
    s.add_atoms(w.tag, w.pos, w.vel, w.mass, w.cutoff, columns=[w.radius])
    if w.harmonic_k:
        s.set_harmonic(w.harmonic_k, rc)
    if c["squeeze"]:
        s.set_deform(0, abi.SOIL_DEFORM_ERATE, c["squeeze"])
    if c["slab"]:
        s.set_boundary([abi.SOIL_BOUNDARY_PERIODIC, abi.SOIL_BOUNDARY_PERIODIC,
                        abi.SOIL_BOUNDARY_SHRINK])
    s.setup()
    if c["phases"]:
        for _ in range(c["steps"]):
            for p in PHASES:
                s.phase(p)
    else:
        s.step(c["steps"])
    a = s.atoms(local_only=True)
    off, idx = s.neighbor()
    room[:len(idx)] = idx
    room[len(idx):] = 0xFFFFFFFF
    s.close()
    return dict(tag=a["tag"], pos=a["pos"], vel=a["vel"], force=a["force"], image=a["image"],
                offsets=off, indices=room)


def run(state):
    c = state["case"]
    if c["kind"] == "run":
        state["sys"].step(c["steps"])
        return _view(state["sys"], state["list"])
    if c["kind"] == "job":
        return _run_job(state["ctx"], c, state["w"], state["list"])
    if c["kind"] == "batch":
        state["batch"].step(c["steps"])
        ends, host = state["ends"], state["np"]
        for i, s in enumerate(state["members"]):
            s.read_local_state(host[0, ends[i]:ends[i + 1]], host[1, ends[i]:ends[i + 1]])
        return dict(pos=state["host"][0], vel=state["host"][1])
    if c["kind"] == "serve":
        srv = state["srv"].server
        ids = [srv.submit(w) for w in state["jobs"]]
        out = []
        for j in ids:
            info = srv.wait(j)
            if info["state"] != "done":
                raise RuntimeError(srv.error(j))
            out.append(srv.result(j))
            srv.release(j)
        return out
    x, out = state["x"], state["out"]
    origin, size, count, lo, box, tilt = state["grid"]
    st = state["ctx"].lib.soil_bin_sort_noalloc(
        state["ctx"].h, x[0].data_ptr(), x[1].data_ptr(), x[2].data_ptr(), c["n"], origin, size,
        count, lo, box, tilt, 0, out[0].data_ptr(), out[1].data_ptr(),
        torch.cuda.current_stream().cuda_stream)
    state["ctx"].check(st, "soil_bin_sort_noalloc")
    return dict(cell=out[0], perm=out[1])


# ---- what a pass cannot do without ---------------------------------------------


def _pairs_per_atom(c):
    """Half-list entries per atom of randomly placed spheres within the pair
    cutoff (mean over the radii), and those in contact."""
    d2 = 1.0 if c["mono"] else 1.0 + 2.0 * (RMAX - RMIN) ** 2 / 12.0
    rho = c["phi"] / (4.0 / 3.0 * math.pi * (0.125 if c["mono"] else MEAN_R3))
    ball = 4.0 / 3.0 * math.pi * rho * 0.5 * d2 ** 1.5
    return ball * (1.0 + SKIN) ** 3, ball


def _step_work(c):
    """Bytes and operations of one step of one atom.  State read and written
    (x, v, f with a consumer; x and v without), mass and radius read; a step
    that must rebuild also writes the list."""
    near, touching = _pairs_per_atom(c)
    b = (3 + 3) * 8 * 2 + 8
    f = 12.0
    if c["k"]:
        b += 3 * 8 * 2 + 8
        f += near * 10.0 + touching * 24.0
    if c["rate"] or c.get("squeeze") or c.get("slab"):
        b += 4 + 4 * near * (1 if c["newton"] else 2)
        f += near * 20.0
    return b, f


def work(case):
    c = case
    if c["kind"] in ("run", "job"):
        b, f = _step_work(c)
        scale = c["n"] * c["steps"]
        extra = 0.0
        if c["kind"] == "job":  # host arrays in (x, v, m, cutoff, radius, tag) and out
            extra = c["n"] * (76 + 24 * 3 + 4 + 12 + 4 + 4 * _pairs_per_atom(c)[0])
        return dict(bytes=scale * b + extra, flops=scale * f)
    if c["kind"] == "binsort":
        return dict(bytes=c["n"] * 32.0, flops=c["n"] * 9.0)
    # boxes log-uniform in [nmin, nmax]: their mean size, half of them sheared
    mean = (c["nmax"] - c["nmin"]) / math.log(c["nmax"] / c["nmin"])
    atoms = mean * (c.get("boxes") or c["jobs"])
    still = _run("", int(mean), 0.375, c["steps"])
    b0, f0 = _step_work(still)
    b1, f1 = _step_work(dict(still, rate=0.1))
    steps = c["steps"] + (15 if c["kind"] == "serve" else 0)
    return dict(bytes=atoms * (steps * 0.5 * (b0 + b1) + (136 if c["kind"] == "serve" else 48)),
                flops=atoms * steps * 0.5 * (f0 + f1))


# ---- the same results in plain torch ---------------------------------------------


class _Sim:
    """One box by the definition: velocity-Verlet with linear repulsion, lists
    good for a displacement of half the skin, wrapped and re-ordered by bin
    when they are renewed.  Everything in float64, atoms in tag order; `order`
    holds the storage order."""

    def __init__(self, c, seed, stream=0):
        self.c = c
        self.x, self.v, self.r = _particles(c, seed, stream)
        self.f = torch.zeros_like(self.x)
        self.cut = self.r if c["mono"] else self.r + 0.5 * SKIN
        self.widest = 2.0 * (0.5 * (1.0 + SKIN) if c["mono"] else float(self.cut.max()))
        self.ghost = self.widest + 2.0 * (SKIN * 0.5)
        self.lo, self.size = np.zeros(3), np.full(3, _side(c))
        self.size0 = self.size.copy()
        self.image = torch.zeros_like(self.x, dtype=torch.int32)
        self.order = torch.arange(c["n"], device="cuda")
        self.at_build = None
        self.tilt = 0.0
        self.step_no = 0
        self.pi = self.pj = None

    def lamda(self, x):
        u = (x - self.t(self.lo)) / self.t(self.size)
        if self.tilt:
            u[:, 0] = (x[:, 0] - self.lo[0] - self.tilt * u[:, 1]) / self.size[0]
        return u

    @staticmethod
    def t(a):
        return torch.tensor(a, dtype=torch.float64, device="cuda")

    def nearest(self, d):
        """Nearest periodic image of difference vectors."""
        if self.c.get("slab"):
            k2 = torch.zeros_like(d[:, 2])
        else:
            k2 = torch.round(d[:, 2] / self.size[2])
        k1 = torch.round(d[:, 1] / self.size[1])
        dx = d[:, 0] - k1 * self.tilt
        k0 = torch.round(dx / self.size[0])
        return torch.stack([dx - k0 * self.size[0], d[:, 1] - k1 * self.size[1],
                            d[:, 2] - k2 * self.size[2]], dim=1)

    def deform(self):
        c, moved = self.c, False
        if c.get("squeeze"):
            old_lo, old = self.lo[0], self.size[0]
            new = self.size0[0] * (1.0 + c["squeeze"] * c["dt"] * self.step_no)
            mid = 0.5 * self.size0[0]
            self.lo[0], self.size[0] = mid - 0.5 * new, new
            self.x[:, 0] = mid + (self.x[:, 0] - (old_lo + 0.5 * old)) * (new / old)
            moved = True
        if c["rate"]:
            ly = self.size[1]
            if self.step_no == 1:
                self.v[:, 0] += c["rate"] * (self.x[:, 1] - 0.5 * ly)
            raw = c["rate"] * c["dt"] * self.step_no * ly
            self.tilt = raw - self.size[0] * round(raw / self.size[0])
            moved = True
        return moved

    def wrap(self):
        """Back into the box; a y crossing in a sheared box moves x by the
        tilt and vx by the drive."""
        axes = 2 if self.c.get("slab") else 3
        u = self.lamda(self.x)
        k = torch.floor(u)
        k[:, axes:] = 0
        self.x -= k * self.t(self.size)
        self.x[:, 0] -= k[:, 1] * self.tilt
        if self.c["rate"]:
            self.v[:, 0] -= k[:, 1] * (self.c["rate"] * self.size[1])
        self.image += k.to(torch.int32)

    def sort(self):
        """Storage order by bin (x slowest), the earlier order kept within a bin."""
        bins = np.maximum(np.floor(self.size / max(1.0, self.widest)), 1.0)
        u = self.lamda(self.x)
        k = torch.floor(u * self.t(bins)).to(torch.int64)
        top = [int(b) + 2 for b in bins]
        key = ((k[:, 0] + 1) * top[1] + k[:, 1] + 1) * top[2] + k[:, 2] + 1
        self.order = self.order[torch.argsort(key[self.order], stable=True)]

    def find_pairs(self):
        """All pairs within the widest cutoff, through a grid of cells at
        least that wide."""
        n, size = self.c["n"], self.size.copy()
        size[0] /= math.sqrt(1.0 + (self.tilt / self.size[1]) ** 2)
        m = [int(s / self.widest) for s in size]
        if min(m) < 3:
            i, j = torch.triu_indices(n, n, 1, device="cuda")
            near = self.nearest(self.x[j] - self.x[i]).square().sum(1) < self.widest ** 2
            return i[near], j[near]
        u = self.lamda(self.x)
        cell = torch.stack([(torch.floor(u[:, d] * m[d]).to(torch.int64)).clamp(0, m[d] - 1)
                            for d in range(3)], dim=1)
        key = (cell[:, 0] * m[1] + cell[:, 1]) * m[2] + cell[:, 2]
        by = torch.argsort(key)
        start = torch.searchsorted(key[by].contiguous(),
                                   torch.arange(m[0] * m[1] * m[2] + 1, device="cuda"))
        ks, xs = cell[by], self.x[by]
        pi, pj = [], []
        offsets = [(a, b, d) for a in (-1, 0, 1) for b in (-1, 0, 1) for d in (-1, 0, 1)
                   if (a, b, d) >= (0, 0, 0)]
        for o in offsets:
            q = ks + torch.tensor(o, device="cuda")
            inside = torch.ones(n, dtype=torch.bool, device="cuda")
            if self.c.get("slab"):
                inside = (q[:, 2] >= 0) & (q[:, 2] < m[2])
            q = q % torch.tensor(m, device="cuda")
            qk = (q[:, 0] * m[1] + q[:, 1]) * m[2] + q[:, 2]
            b, e = start[qk], start[qk + 1]
            if o == (0, 0, 0):
                b = torch.arange(n, device="cuda") + 1
            cnt = torch.where(inside, (e - b).clamp(min=0), torch.zeros_like(b))
            i = torch.repeat_interleave(torch.arange(n, device="cuda"), cnt)
            first = torch.cumsum(cnt, 0) - cnt
            j = torch.arange(i.numel(), device="cuda") - first[i] + b[i]
            near = self.nearest(xs[j] - xs[i]).square().sum(1) < self.widest ** 2
            pi.append(by[i[near]])
            pj.append(by[j[near]])
        return torch.cat(pi), torch.cat(pj)

    def forces(self):
        if not self.c["k"]:
            return
        d = self.nearest(self.x[self.pj] - self.x[self.pi])
        reach = self.r[self.pi] + self.r[self.pj]
        r2 = d.square().sum(1)
        hit = (r2 < reach * reach) & (r2 > 0)
        i, j, d, dist = self.pi[hit], self.pj[hit], d[hit], r2[hit].sqrt()
        push = (self.c["k"] * (reach[hit] - dist) / dist)[:, None] * d
        if not self.c["newton"]:  # full lists: a pair with no image in it is visited twice
            same = (d - (self.x[j] - self.x[i])).abs().amax(1) < 0.25 * self.size.min()
            push = push * torch.where(same, 2.0, 1.0)[:, None].to(torch.float64)
        self.f = torch.zeros_like(self.x).index_add_(0, i, -push).index_add_(0, j, push)

    def step(self):
        dt = self.c["dt"]
        self.step_no += 1
        moved = self.deform()
        self.v = self.v + 0.5 * dt * self.f
        self.x = self.x + dt * self.v
        due = moved or self.at_build is None
        if not due:
            far = self.nearest(self.x - self.at_build).square().sum(1).max()
            due = float(far) > (0.5 * SKIN) ** 2
        if self.c.get("slab"):
            z = self.x[:, 2]
            self.lo[2] = float(z.min()) - self.ghost
            self.size[2] = float(z.max()) + self.ghost - self.lo[2]
        if due:
            self.wrap()
            self.sort()
            if self.c["k"]:
                self.pi, self.pj = self.find_pairs()
            self.at_build = self.x.clone()
        self.forces()
        self.v = self.v + 0.5 * dt * self.f

    def advance(self, steps):
        for _ in range(steps):
            self.step()
        return [a[self.order] for a in (self.x, self.v, self.f)]


def exact(case, seed):
    c = case
    if c["kind"] == "run":
        x, v, f = _Sim(c, seed).advance(c["steps"])
        out = {k: x[:, d].contiguous() for d, k in enumerate(("x", "y", "z"))}
        out.update({k: v[:, d].contiguous() for d, k in enumerate(("vx", "vy", "vz"))})
        out.update({k: f[:, d].contiguous() for d, k in enumerate(("fx", "fy", "fz"))})
        return dict(out, tag=None, offsets=None, indices=None)
    if c["kind"] == "job":
        x, v, f = _Sim(c, seed).advance(c["steps"])
        return dict(tag=None, pos=x, vel=v, force=f, image=None, offsets=None, indices=None)
    if c["kind"] == "batch":
        if c["boxes"] * c["steps"] > 2500:  # a loop over the boxes would take too long
            return None
        got = [_Sim(b, seed, i).advance(b["steps"]) for i, b in enumerate(_boxes(c))]
        return dict(pos=torch.cat([g[0] for g in got]), vel=torch.cat([g[1] for g in got]))
    if c["kind"] == "serve":
        out = []
        for i, b in enumerate(_boxes(c)):
            x, v, _ = _Sim(b, seed, i).advance(b["steps"])
            out.append(dict(tag=None, pos=x, vel=v, image=None))
        return out
    return None
