"""Performance cases of the reaction-diffusion backend.

A case is a plain dict; `prepare` builds the simulation a user's program holds (a
configured, initialised Solver or Batch with its field and agents on the GPU), `run`
is one pass through the public entry points, `work` what the pass cannot do without,
and `exact` the same pass in 64 bits with plain torch.  Sizes restate the benchmark
workloads (workloads.py), the example driver's settings and the test meshes.

kind   step     `steps` solver steps with the agents where they are (the inner loop
                of a simulation between two phenotype updates)
       moved    the agents were moved on the device, so the step rebuilds the ballot
                (the loop of a simulation with motile cells)
       image    agent positions come from the host and the whole field, the
                internalized amounts and the counts go back (the loop of a host
                program that writes images and keeps its agents on the CPU)
       batch    many uneven domains stepped together (parameter studies, serving)
"""
import math

import numpy as np
import torch

import physicore_gb300 as pcg

VOXEL, DT = 20, 0.01

_streams = {}


def _stream():
    """The one stream a program queues all its simulations on."""
    dev = torch.cuda.current_device()
    if dev not in _streams:
        _streams[dev] = torch.cuda.Stream()
    return _streams[dev]


def _case(name, kind, prec, nx, ny, nz, S, agents, steps=1, faces="x", interior=0, bulk="none", cluster=0.0,
          internalized=True, mass_check=False):
    """nz == 0: a 2-D mesh; ny == 0 as well: 1-D.  cluster: sigma (um) of a Gaussian
    agent cluster at the centre, 0 for uniform agents."""
    return dict(name=name, kind=kind, prec=prec, nx=nx, ny=ny, nz=nz, S=S, agents=agents, steps=steps, faces=faces,
                interior=interior, bulk=bulk, cluster=cluster, internalized=internalized, mass_check=mass_check)


def _batch(name, prec, domains, side_lo, side_hi, S_hi, agents_hi, sizes_seed, steps=1, moved=False):
    return dict(name=name, kind="batch", prec=prec, domains=domains, side_lo=side_lo, side_hi=side_hi, S_hi=S_hi,
                agents_hi=agents_hi, sizes_seed=sizes_seed, steps=steps, moved=moved)


def listed():
    return [
        # the example driver's 2-D tissue slab at the reference's own precision: ten
        # steps of one small mesh, all launch latency
        _case("slab_2d_fp64", "step", "fp64", 120, 120, 0, 3, 100, steps=10, faces="all"),
        # a small 3-D mesh of the kind tests and first experiments use, one step a call
        _case("small_3d_fp32", "step", "fp32", 48, 40, 36, 2, 1000),
        # the reference's own benchmark mesh and precision
        _case("plain_100_fp64", "step", "fp64", 100, 100, 100, 1, 1000, faces="all"),
        # odd sides and an odd substrate count, interior nodes and uniform bulk rates
        _case("ragged_fp32", "step", "fp32", 97, 131, 61, 5, 20000, faces="all", interior=500, bulk="uniform"),
        # an ordinary tissue at the plugin's default (64-bit) precision
        _case("tissue_fp64", "step", "fp64", 160, 144, 128, 3, 50000, interior=1000),
        # a wide 2-D culture with bulk rates per voxel
        _case("sheet_2d_fp32", "step", "fp32", 1000, 800, 0, 3, 40000, faces="all", bulk="voxel"),
        # oxygen alone on a large mesh, motile cells
        _case("oxygen_fp32", "moved", "fp32", 320, 320, 256, 1, 200000, faces="all"),
        # the headline workload (its step runs with the per-step mass check)
        _case("large_320_fp32", "step", "fp32", 320, 320, 320, 8, 1000000, interior=10000, mass_check=True),
        # a tumour: 4M cells in a Gaussian cluster, moved every step
        _case("dense_200_fp32", "moved", "fp32", 200, 200, 200, 4, 4000000, faces="none", cluster=200.0),
        # a signalling network of many substrates
        _case("signals_fp32", "step", "fp32", 96, 80, 64, 20, 30000),
        # a host program: positions in, planar 64-bit image and amounts out
        _case("image_fp32", "image", "fp32", 160, 160, 128, 4, 20000),
        # uneven independent domains of a parameter study
        _batch("batch_48_fp32", "fp32", 48, 32, 160, 6, 50000, 3),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the same ranges: sides 8-320 (2-D to 1000), 1-24 substrates,
    both precisions, every kind and option."""
    kind = rng.choice(["step", "step", "step", "moved", "image", "batch"])
    prec = rng.choice(["fp32", "fp32", "fp64"])
    if kind == "batch":
        c = _batch("", prec, rng.randint(4, 48), 16, rng.choice([64, 128, 160]), rng.randint(1, 8),
                   int(_log(rng, 200, 50000)), rng.randrange(1 << 20), steps=rng.randint(1, 3),
                   moved=rng.random() < 0.4)
        while _batch_points(c) > (6e7 if prec == "fp32" else 1.5e7):
            c["domains"] = max(2, c["domains"] // 2)
            c["side_hi"] = max(24, int(c["side_hi"] * 0.8))
    else:
        S = rng.choice([1, 1, 2, 3, 3, 4, 5, 6, 7, 8, 8, int(_log(rng, 9, 24))])
        cap = {"fp32": 1.2e8, "fp64": 1.5e7}[prec]
        if kind == "image":
            cap = 1.5e7
        if rng.random() < 0.25:  # 2-D
            nx, ny, nz = int(_log(rng, 20, 1000)), int(_log(rng, 20, 800)), 0
            nx = min(nx, int(200 * 1024 / (S * (4 if prec == "fp32" else 8))))
        else:
            nx, ny, nz = (int(_log(rng, 8, 320)) for _ in range(3))
        while nx * ny * max(nz, 1) * S > cap:
            nx, ny, nz = max(8, int(nx * 0.8)), max(8, int(ny * 0.8)), int(nz * 0.8)
        V = nx * ny * max(nz, 1)
        agents = int(_log(rng, 50, max(60, min(V / 2, 1e6))))
        steps = rng.choice([1, 1, 4, 10]) if kind == "step" and V * S < 1e6 else 1
        bulk = rng.choice(["none", "none", "none", "uniform", "voxel"])
        if V * S > 6e6 and bulk == "voxel":
            bulk = "uniform"
        c = _case("", kind, prec, nx, ny, nz, S, agents, steps=steps, faces=rng.choice(["x", "all", "none"]),
                  interior=int(V * 3e-4) if rng.random() < 0.5 else 0, bulk=bulk,
                  cluster=0.0 if rng.random() < 0.7 else max(40.0, 3.0 * nx), internalized=rng.random() < 0.8,
                  mass_check=rng.random() < 0.2)
    del c["name"]
    return c


def _batch_sizes(case):
    """The domains (sides, substrates, agents) of a batch: log-uniform sides and agents."""
    r = np.random.Generator(np.random.PCG64(case["sizes_seed"]))
    out = []
    for _ in range(case["domains"]):
        sides = tuple(int(round(v)) for v in np.exp(r.uniform(math.log(case["side_lo"]), math.log(case["side_hi"]), 3)))
        S = int(r.integers(1, case["S_hi"] + 1))
        A = int(round(math.exp(r.uniform(math.log(100), math.log(case["agents_hi"])))))
        out.append((sides, S, A))
    return out


def _batch_points(case):
    return sum(s[0] * s[1] * s[2] * S for s, S, _ in _batch_sizes(case))


class _Inputs:
    """The inputs of one domain, from the seed alone (torch's generator on the GPU)."""

    def __init__(self, case, seed, sides=None, S=None, A=None):
        g = torch.Generator(device="cuda")
        g.manual_seed(int(seed))

        def rand(*shape, dtype=torch.float64):
            return torch.rand(*shape, generator=g, device="cuda", dtype=dtype)

        nx, ny, nz = sides or (case["nx"], case["ny"], case["nz"])
        self.dims = 1 if ny == 0 else 2 if nz == 0 else 3
        self.n = (nx, max(ny, 1), max(nz, 1))
        self.S, self.A = S or case["S"], A if A is not None else case["agents"]
        S, A, dims = self.S, self.A, self.dims
        self.w = 4 if case["prec"] == "fp32" else 8
        u = rand(2, S).cpu().numpy()
        self.D = 10.0 * (1e4 ** u[0])           # log-uniform [10, 1e5] um^2/min
        self.decay = 1e-4 * (1e4 ** u[1])       # log-uniform [1e-4, 1] 1/min
        self.field = rand(self.n[2], self.n[1], self.n[0], S, dtype=torch.float32 if self.w == 4 else torch.float64)
        faces = case.get("faces", "x")
        which = {"x": 1, "all": dims, "none": 0}[faces]
        fv = rand(3, 2, S).cpu().numpy()
        self.faces = [(a, side, fv[a, side]) for a in range(which) for side in (0, 1)]
        V = self.n[0] * self.n[1] * self.n[2]
        K = case.get("interior", int(round(V * 3e-4)))
        self.interior = None
        if K:
            lin = torch.unique((rand(K) * V).long().clamp_(max=V - 1))
            vox = torch.stack([lin % self.n[0], (lin // self.n[0]) % self.n[1], lin // (self.n[0] * self.n[1])], 1)
            self.interior = (lin, vox[:, :dims].cpu().numpy().astype(np.uint64), rand(lin.numel(), S))
        self.bulk = case.get("bulk", "none")
        if self.bulk != "none":
            shape = (3, S) if self.bulk == "uniform" else (3, S, self.n[2], self.n[1], self.n[0])
            self.bulk_tables = rand(*shape)
        ext = torch.tensor([v * float(VOXEL) for v in self.n[:dims]], dtype=torch.float64, device="cuda")
        top = ext * (1 - 1e-12)  # inside the last voxel, also after the division by its edge

        def positions():
            if case.get("cluster", 0.0) > 0:
                p = torch.randn(A, dims, generator=g, device="cuda", dtype=torch.float64) * case["cluster"] + ext / 2
                return torch.minimum(p.clamp_(min=0.0), top)
            return torch.minimum(rand(A, dims) * ext, top)

        self.pos, self.pos2 = positions(), positions()
        self.sec, self.upt = rand(A, S), 0.5 * rand(A, S)
        self.vol = 2494.0
        self.internalized = case.get("internalized", True)

    def solver(self, prec):
        """The user's setup: describe, initialise, field written in place on the device."""
        s = pcg.Solver(pcg.FP32 if prec == "fp32" else pcg.FP64)
        ext = [v * VOXEL if a < self.dims else 0 for a, v in enumerate(self.n)]
        s.set_mesh(self.dims, (0, 0, 0), tuple(ext), (VOXEL,) * 3)
        s.set_substrates(DT, self.D, self.decay, np.zeros(self.S))
        for axis, side, values in self.faces:
            s.set_dirichlet_boundary(axis, side, values, np.ones(self.S, np.uint8))
        if self.interior is not None:
            _, vox, values = self.interior
            s.set_dirichlet_interior(vox, values.cpu().numpy(), np.ones(values.shape, np.uint8))
        if self.bulk != "none":
            t = self.bulk_tables.cpu().numpy()
            s.set_bulk(pcg.BULK_UNIFORM if self.bulk == "uniform" else pcg.BULK_PER_VOXEL, t[0], t[1], t[2])
        s.set_stream(_stream().cuda_stream)
        s.initialize()
        if self.A:
            h = [t.cpu().numpy() for t in (self.pos, self.sec, self.upt)]
            s.set_agents(h[0], h[1], np.ones((self.A, self.S)), h[2], np.zeros((self.A, self.S)),
                         np.full(self.A, self.vol), np.ones(self.A, np.uint8),
                         compute_internalized=self.internalized)
        s.synchronize()
        view = _field_view(s)
        view.copy_(self.field.reshape(view.shape))
        torch.cuda.synchronize()
        return s, view

    # ---- the same in 64 bits

    def sweep(self, f, axis):
        g = f.movedim(2 - axis, 0)
        n = g.shape[0]
        D, decay = (torch.tensor(v, dtype=torch.float64, device="cuda") for v in (self.D, self.decay))
        r = DT * D / float(VOXEL * VOXEL)
        diag = [1 + decay * DT / self.dims + 2 * r - (r if i in (0, n - 1) else 0) for i in range(n)]
        cp = []
        for i in range(n):
            m = diag[i] - (r * cp[i - 1] if i else 0)
            g[i] = ((g[i] + r * g[i - 1]) if i else g[i]) / m
            cp.append(r / m)
        for i in range(n - 2, -1, -1):
            g[i] += cp[i] * g[i + 1]

    def step(self, f, amounts, pos):
        """One step of the field f [nz, ny, nx, S] and the amounts [A, S], in place;
        returns the agents per voxel."""
        for a in range(self.dims):
            self.sweep(f, a)
        for axis, side, values in self.faces:
            f.select(2 - axis, -1 if side else 0).copy_(torch.tensor(values, device="cuda"))
        flat = f.view(-1, self.S)
        if self.interior is not None:
            flat[self.interior[0]] = self.interior[2]
        if self.bulk != "none":
            t = self.bulk_tables if self.bulk == "uniform" else self.bulk_tables.permute(0, 2, 3, 4, 1)
            f.copy_((f + DT * t[0] * t[2]) / (1 + DT * (t[1] + t[0])))
        V, Vv = flat.shape[0], float(VOXEL) ** 3
        if not self.A:
            return torch.zeros(V, dtype=torch.int64, device="cuda")
        last = torch.tensor(self.n[:self.dims], device="cuda") - 1
        idx = torch.minimum((pos / VOXEL).long(), last)
        vox = idx[:, 0]
        for a, stride in ((1, self.n[0]), (2, self.n[0] * self.n[1])):
            if a < self.dims:
                vox = vox + stride * idx[:, a]
        num, den = self.sec * (DT * self.vol / Vv), (self.upt + self.sec) * (DT * self.vol / Vv)
        occupied, where, count = torch.unique(vox, return_inverse=True, return_counts=True)
        zero = torch.zeros(occupied.numel(), self.S, dtype=torch.float64, device="cuda")
        sn, sd = zero.index_add(0, where, num), zero.index_add(0, where, den)
        old = flat[occupied]
        new = (old + sn) / (1 + sd)
        flat[occupied] = new
        if self.internalized:
            if int(count.max()) == 1:
                amounts += (Vv * (old - new))[where]
            else:
                amounts -= Vv * (num - new[where] * den)
        counts = torch.zeros(V, dtype=torch.int64, device="cuda")
        counts[occupied] = count
        return counts


class _Array:
    """A solver's device memory as an array object that torch views without a copy; the
    view keeps the solver alive."""

    def __init__(self, owner, ptr, shape, strides, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, strides=strides, typestr=typestr, data=(ptr, False), version=3)


def _field_view(s):
    """The solver's device field as a tensor [nz, ny, nx * S] (rows padded to the pitch)."""
    ptr, w, pitch = s.field_device()
    nx, ny, nz = s.grid
    return torch.as_tensor(_Array(s, ptr, (nz, ny, nx * s.S), (ny * pitch * w, pitch * w, w), "<f%d" % w), device="cuda")


class _State:
    pass


def _domain_inputs(case, seed):
    for i, (sides, S, A) in enumerate(_batch_sizes(case)):
        yield _Inputs(case, (int(seed) * 1000003 + i) % (1 << 62), sides, S, A)


def prepare(case, seed):
    st = _State()
    st.case = case
    if case["kind"] == "batch":
        pairs = [x.solver(case["prec"]) for x in _domain_inputs(case, seed)]
        st.solvers, st.views = [p[0] for p in pairs], [p[1] for p in pairs]
        st.batch = pcg.Batch(st.solvers)
        st.batch.prepare()
        return st
    x = _Inputs(case, seed)
    st.solver, st.view = x.solver(case["prec"])
    if case["mass_check"]:
        st.solver.set_mass_check(True)
    if case["kind"] == "image":
        st.pos = x.pos2.cpu().numpy()
        nx, ny, nz = st.solver.grid
        st.image = torch.empty((x.S, nz, ny, nx), dtype=torch.float64, pin_memory=True).numpy()
    torch.cuda.synchronize()
    return st


def run(st):
    case = st.case
    if case["kind"] == "batch":
        if case["moved"]:
            for s in st.solvers:
                s.recompute_positional_data()
        st.batch.solve(case["steps"])
        return st.views
    s = st.solver
    if case["kind"] == "image":
        s.update_agents(positions=st.pos)
        s.recompute_positional_data()
        s.solve(case["steps"])
        s.get_field(pcg.LAYOUT_PLANAR, np.float64, out=st.image)
        return [st.image, s.get_internalized(), s.get_counts().view(np.int32)]
    if case["kind"] == "moved":
        s.recompute_positional_data()
    s.solve(case["steps"])
    return st.view


def _work(case, dims, V, S, A):
    w = 4 if case["prec"] == "fp32" else 8
    moved = case["kind"] in ("moved", "image") or case.get("moved", False)
    internalized = case.get("internalized", True)
    b = 2.0 * V * S * w + A * (8 + 3 * S * w + (16 * S if internalized else 0)) + (A * (8 * dims + 1) if moved else 0)
    if case.get("bulk", "none") == "voxel":
        b += 3.0 * V * S * w
    if case["kind"] == "image":
        b += 8.0 * V * S + 4.0 * V + 8.0 * A * S
    f = case["steps"] * (5.0 * dims * V * S + (7.0 * V * S if case.get("bulk", "none") != "none" else 0) + 12.0 * A * S)
    return b, f


def work(case):
    if case["kind"] == "batch":
        parts = [_work(case, 3, s[0] * s[1] * s[2], S, A) for s, S, A in _batch_sizes(case)]
    else:
        dims = 1 if case["ny"] == 0 else 2 if case["nz"] == 0 else 3
        parts = [_work(case, dims, case["nx"] * max(case["ny"], 1) * max(case["nz"], 1), case["S"], case["agents"])]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


def exact(case, seed):
    if case["kind"] == "batch":
        out = []
        for x in _domain_inputs(case, seed):
            f, amounts = x.field.double(), torch.zeros(x.A, x.S, dtype=torch.float64, device="cuda")
            for _ in range(case["steps"]):
                x.step(f, amounts, x.pos)
            out.append(f.reshape(x.n[2], x.n[1], x.n[0] * x.S))
        return out
    x = _Inputs(case, seed)
    f, amounts = x.field.double(), torch.zeros(x.A, x.S, dtype=torch.float64, device="cuda")
    image = case["kind"] == "image"
    for _ in range(case["steps"]):
        counts = x.step(f, amounts, x.pos2 if image else x.pos)
    if image:
        return [f.permute(3, 0, 1, 2).contiguous(), amounts, counts.reshape(x.n[2], x.n[1], x.n[0])]
    return f.reshape(x.n[2], x.n[1], x.n[0] * x.S)
