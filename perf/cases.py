"""Performance cases of the cell-step framework: what its users run, at the sizes they run it.

Every case is one pass of a program's main loop.  A simulation case uploads a
state that is on the GPU, advances it a few steps and takes the new state
back on the GPU (``Simulation.set_state_device``, ``take_step`` and the C
ABI's ``tecs_sim_download_device``).  The ensemble case admits a batch of
simulations to the multi-simulation engine, steps them together, downloads
each one and retires them, as the batched and served forms do.

``exact`` integrates the same equations in 64 bits with plain torch.
"""
import ctypes
import math

import numpy as np
import torch

import tecs_gb300 as tg
from tecs_gb300.engine import Engine, bins_needed

DT = 0.05
# the spring constants and the cutoff of the framework's default description
K_REP, R_REP, K_ADH, R_ADH, K_POL = 2.0, 0.7, 0.5, 0.8, 0.2
CUTOFF = 1.0
GABRIEL = 0.8
SEED = 2807


def _sim(name, shape, n, steps, finder="binned_gabriel", integrator="heun", law="spring", com=False, division=0.0):
    case = dict(kind="simulation", shape=shape, n=n, steps=steps, finder=finder, integrator=integrator, law=law,
                com=com, division=division)
    return dict(case, name=name) if name else case


def listed():
    return [
        # the smallest simulations: a thousand cells, where a step is launches and latency
        _sim("small_allpairs_1k", "ball", 1000, 100, finder="binned_all_pairs", integrator="euler"),
        # the default configuration's finder and integrator, as the spring programs use them
        _sim("default_naive_2k", "ball", 2003, 20, finder="naive_all_pairs"),
        # the example program of the naive Delaunay finder: a few hundred cells in a ball
        _sim("naive_delaunay_400", "ball", 400, 1, finder="naive_delaunay", integrator="euler"),
        # an epithelial sheet with apical-basal polarity, wrapped around a sphere
        _sim("sheet_polarity_100k", "sheet", 100_000, 3, law="polarity"),
        # a two-dimensional culture
        _sim("disk_gabriel_60k", "disk", 60_013, 10, integrator="euler"),
        # a compact tissue: the packing that the relaxed initialisers give at spacing 0.8
        _sim("packed_gabriel_200k", "packed", 199_999, 5),
        # a growing spheroid at full size: centre-of-mass fix and division
        _sim("spheroid_1m", "ball", 1_000_000, 10, com=True, division=1e-4),
        # overlapping cells without pruning, one evaluation a step
        _sim("allpairs_300k", "ball", 300_007, 10, finder="binned_all_pairs", integrator="euler"),
        # a batch of independent simulations, half Gabriel and half all-pairs
        dict(name="ensemble_32", kind="ensemble", sims=32, lo=500, hi=200_000, steps=20),
        # Delaunay neighbours past the naive finder's size, in the plane and in space
        _sim("delaunay_disk_30k", "disk", 30_011, 1, finder="delaunay"),
        _sim("delaunay_ball_40k", "ball", 40_009, 1, finder="delaunay", integrator="euler"),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    integrator = rng.choice(["euler", "heun"])
    kind = rng.choice(["binned", "binned", "binned", "sheet", "packed", "small", "naive", "delaunay", "ensemble"])
    if kind == "binned":
        com = rng.random() < 0.5
        return _sim(None, rng.choice(["ball", "ball", "disk"]), size(2000, 1_000_000), rng.randint(2, 10),
                    finder=rng.choice(["binned_gabriel", "binned_all_pairs"]), integrator=integrator, com=com,
                    division=rng.choice([0.0, 1e-4]))
    if kind == "sheet":
        return _sim(None, "sheet", size(1000, 200_000), rng.randint(1, 3), integrator=integrator, law="polarity")
    if kind == "packed":
        return _sim(None, "packed", size(1000, 300_000), rng.randint(2, 5), integrator=integrator)
    if kind == "small":
        return _sim(None, "ball", size(100, 4000), rng.randint(10, 100),
                    finder=rng.choice(["binned_gabriel", "binned_all_pairs"]), integrator=integrator)
    if kind == "naive":
        finder = rng.choice(["naive_all_pairs", "naive_gabriel"])
        return _sim(None, rng.choice(["ball", "disk"]), size(100, 4000), rng.randint(2, 20), finder=finder,
                    integrator=integrator)
    if kind == "delaunay":
        shape = rng.choice(["ball", "disk"])
        return _sim(None, shape, size(1000, 30_000), 1, finder="delaunay", integrator=integrator)
    return dict(kind="ensemble", sims=rng.randint(4, 32), lo=500, hi=rng.randint(5000, 150_000),
                steps=rng.randint(5, 20))


# ---------------------------------------------------------------------------
# inputs, made on the GPU from the seed


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _directions(n, g):
    d = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    return d / d.norm(dim=1, keepdim=True)


def _ball(n, g):
    """Uniform in a ball at one cell per unit volume."""
    radius = (3.0 * n / (4.0 * math.pi)) ** (1.0 / 3.0)
    r = radius * torch.rand(n, 1, generator=g, device="cuda", dtype=torch.float64) ** (1.0 / 3.0)
    return (_directions(n, g) * r).float()


def _disk(n, g):
    """Uniform in a disk at one cell per unit area."""
    u = torch.rand(n, 2, generator=g, device="cuda", dtype=torch.float64)
    r, t = torch.sqrt(u[:, 0] * n / math.pi), u[:, 1] * 2.0 * math.pi
    return torch.stack([r * torch.cos(t), r * torch.sin(t)], 1).float()


def _packed(n, g, spacing=0.84, jitter=0.06):
    """A ball of n cells on a jittered face-centred lattice: 2.39 cells per
    unit volume, the density of the relaxed initialisers at spacing 0.8."""
    side = int((4.0 * n) ** (1.0 / 3.0)) + 6
    k = torch.arange(side, device="cuda") - side // 2
    c = torch.stack(torch.meshgrid(k, k, k, indexing="ij"), -1).reshape(-1, 3)
    c = c[(c.sum(1) % 2) == 0].double() * (spacing / math.sqrt(2.0))
    c = c[torch.argsort(c.norm(dim=1), stable=True)[:n]]
    c = c + jitter * torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    return c[torch.randperm(n, generator=g, device="cuda")].float()


def _sheet(n, g):
    """A jittered spherical shell with outward polarities."""
    radius = math.sqrt(n / (4.0 * math.pi)) * 0.8
    jitter = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    x = (_directions(n, g) * radius + 0.02 * jitter).float()
    xd = x.double()
    noise = 0.1 * torch.randn(n, 2, generator=g, device="cuda", dtype=torch.float64)
    theta = torch.acos((xd[:, 2] / xd.norm(dim=1)).clamp(-1, 1)) + noise[:, 0]
    phi = torch.atan2(xd[:, 1], xd[:, 0]) + noise[:, 1]
    return x, torch.stack([theta, phi], 1).float()


def _inputs(case, seed):
    g = _generator(seed)
    if case["shape"] == "sheet":
        return _sheet(case["n"], g)
    return {"ball": _ball, "disk": _disk, "packed": _packed}[case["shape"]](case["n"], g), None


def _settings(x, capacity):
    half = float(math.ceil(float(x.abs().max()) + 2.0))
    pf = tg.PairFinderSettings(min_bounds=(-half,) * 3, max_bounds=(half,) * 3)
    return tg.Settings(agent_count=len(x), capacity=capacity, cutoff_distance=CUTOFF, seed=SEED,
                       pair_finder_settings=pf)


def _capacity(case):
    # a growing tissue keeps room for its daughters
    return int(case["n"] * 1.05) + 64 if case["division"] else case["n"]


def _members(case, seed):
    """The batch: cell counts log-uniform, spring constants of their own, half of them with the Gabriel finder."""
    rng = np.random.default_rng(int(seed) + 17)
    counts = np.exp(np.linspace(math.log(case["lo"]), math.log(case["hi"]), case["sims"])).astype(int)
    k_rep, k_adh = rng.uniform(1.5, 2.5, case["sims"]), rng.uniform(0.3, 0.7, case["sims"])
    g = _generator(seed)
    return [(_ball(int(n) + k, g), "binned_gabriel" if k % 2 else "binned_all_pairs",
             tg.Spring2R(k_rep=float(k_rep[k]), k_adh=float(k_adh[k]))) for k, n in enumerate(counts)]


def prepare(case, seed):
    if case["kind"] == "ensemble":
        descs, states = [], []
        for x, finder, force in _members(case, seed):
            descs.append(tg.make_desc(_settings(x, len(x)), pair_finder=finder, integrator="heun", force=force))
            states.append(x.cpu().numpy())
        cells = sum(len(x) for x in states)
        engine = Engine(cell_capacity=cells + 1024, bin_capacity=sum(bins_needed(d) for d in descs) + 1024,
                        max_sims=len(descs) + 8)
        return dict(case=case, engine=engine, descs=descs, states=states)
    x, p = _inputs(case, seed)
    capacity = _capacity(case)
    polarity = p is not None
    sim = tg.Simulation(
        _settings(x, capacity), dims=x.shape[1], pair_finder=case["finder"], integrator=case["integrator"],
        com_fixer="global" if case["com"] else None, polarity=polarity,
        force=tg.PolaritySpring(k_pol=K_POL) if case["law"] == "polarity" else tg.Spring2R(),
        division=tg.Division(probability=case["division"]))
    out = torch.empty(capacity, x.shape[1], device="cuda")
    out_p = torch.empty(capacity, 2, device="cuda") if polarity else None
    torch.cuda.synchronize()  # the simulation reads the state on its own stream
    return dict(case=case, sim=sim, x=x, p=p, out=out, out_p=out_p)


def run(state):
    case = state["case"]
    if case["kind"] == "ensemble":
        engine = state["engine"]
        slots = [engine.add(d, x) for d, x in zip(state["descs"], state["states"])]
        engine.step(DT, case["steps"])
        results = [engine.download(s)[0] for s in slots]
        for s in slots:
            engine.remove(s)
        return results
    sim, x, p, out, out_p = (state[k] for k in ("sim", "x", "p", "out", "out_p"))
    sim.set_state_device(x.data_ptr(), None if p is None else p.data_ptr(), len(x))
    sim.take_step(DT, case["steps"])
    lib, count = tg.load(), ctypes.c_uint()
    if lib.tecs_sim_download_device(sim._h, ctypes.c_void_p(out.data_ptr()),
                                    None if p is None else ctypes.c_void_p(out_p.data_ptr()), ctypes.byref(count)):
        raise tg.TecsError(lib.tecs_last_error().decode())
    n = count.value
    return {"cells": n, "x": out[:n], "p": None if p is None else out_p[:n]}


# ---------------------------------------------------------------------------
# the work of a pass


def work(case):
    """The state is read and written once a pass (between the steps it may stay on the chip); the operations of
    each force evaluation are the distance tests, the witness tests and the accepted pairs' forces."""
    if case["kind"] == "ensemble":
        counts = np.exp(np.linspace(math.log(case["lo"]), math.log(case["hi"]), case["sims"])).astype(int)
        n, evaluations, dims, finder, law, density = float(counts.sum()), 2, 3, "binned_gabriel", "spring", 1.0
    else:
        n, finder, law = case["n"], case["finder"], case["law"]
        evaluations = 2 if case["integrator"] == "heun" else 1
        dims = 2 if case["shape"] == "disk" else 3
        density = {"ball": 1.0, "disk": 1.0, "packed": 2.39, "sheet": 0.5}[case["shape"]]
    near = {"sheet": 5.0}.get(case.get("shape"), density * (math.pi if dims == 2 else 4.19))
    if finder == "naive_delaunay":
        flops = n * near * n * 60.0  # every third point of every near pair has its own sphere
    elif finder == "delaunay":
        flops = n * (6 if dims == 2 else 24) * 200.0  # the simplices around each cell
    else:
        candidates = n if finder.startswith("naive") else density * 3.0 ** dims
        flops = n * (candidates * 8.0 + near * 25.0)
        if finder.endswith("gabriel"):
            flops += n * near * near * 8.0
        if law == "polarity":
            flops += n * near * 250.0
    width = 4.0 * dims + (8.0 if law == "polarity" else 0.0)
    passes = evaluations * case["steps"]
    return {"bytes": 2.0 * n * width, "flops": flops * passes}


# ---------------------------------------------------------------------------
# the same equations in 64 bits


def _f32(v):
    return float(np.float32(v))


class _Bins:
    """Cells sorted by bin, as a step's grid holds them: the positions may move on afterwards."""

    def __init__(self, x, half):
        self.dims = x.shape[1]
        self.half = half
        self.ext = int(math.ceil(2.0 * half / CUTOFF))
        self.cell = self.coords(x)
        key = self.flat(self.cell)
        self.order = torch.argsort(key, stable=True)
        bins = torch.arange(self.ext**self.dims + 1, device=x.device)
        self.off = torch.searchsorted(key[self.order].contiguous(), bins)

    def coords(self, x):
        return torch.trunc((x + self.half) / CUTOFF).clamp(0, self.ext - 1).long()

    def flat(self, c):
        b = c[:, 0] + c[:, 1] * self.ext
        return b + c[:, 2] * self.ext**2 if self.dims == 3 else b

    def pairs(self, x):
        """In-cutoff (i, j) over the 3^dims bins around each cell's present position, sorted by i."""
        home = self.coords(x)
        found = []
        lo_x, hi_x = (home[:, 0] - 1).clamp(min=0), (home[:, 0] + 1).clamp(max=self.ext - 1)
        for dz in (-1, 0, 1) if self.dims == 3 else (0,):
            for dy in (-1, 0, 1):
                row = home.clone()
                row[:, 1] += dy
                ok = (row[:, 1] >= 0) & (row[:, 1] < self.ext)
                if self.dims == 3:
                    row[:, 2] += dz
                    ok &= (row[:, 2] >= 0) & (row[:, 2] < self.ext)
                row = row.clamp(0, self.ext - 1)
                row[:, 0] = lo_x
                lo = self.off[self.flat(row)]
                row[:, 0] = hi_x
                count = torch.where(ok, self.off[self.flat(row) + 1] - lo, 0)
                i = torch.repeat_interleave(torch.arange(len(x), device=x.device), count)
                start = torch.cumsum(count, 0) - count
                j = self.order[lo[i] + torch.arange(len(i), device=x.device) - start[i]]
                near = ((x[i] - x[j]).square().sum(1) < CUTOFF * CUTOFF) & (i != j)
                found.append(torch.stack([i[near], j[near]], 1))
        found = torch.cat(found)
        found = found[torch.argsort(found[:, 0], stable=True)]
        return found[:, 0], found[:, 1]


def _gabriel(x, bins, i, j):
    """The pairs without a witness in the ball around their midpoint (for binned finders: in the bins it touches)."""
    count = torch.bincount(i, minlength=len(x))
    first = torch.cumsum(count, 0) - count
    keep = torch.ones(len(i), dtype=torch.bool, device=x.device)
    c = _f32(GABRIEL)
    for a in range(0, len(i), 1 << 21):
        pi, pj = i[a:a + (1 << 21)], j[a:a + (1 << 21)]
        m = 0.5 * (x[pi] + x[pj])
        rsq = (x[pi] - x[pj]).square().sum(1) * (c * c * 0.25)
        r = torch.sqrt(rsq)[:, None]
        w = torch.repeat_interleave(torch.arange(len(pi), device=x.device), count[pi])
        start = torch.cumsum(count[pi], 0) - count[pi]
        k = j[first[pi][w] + torch.arange(len(w), device=x.device) - start[w]]
        hit = ((x[k] - m[w]).square().sum(1) < rsq[w]) & (k != pj[w])
        if bins is not None:
            lo = torch.floor((m - r + bins.half) / CUTOFF).clamp(0, bins.ext - 1).long()
            hi = torch.floor((m + r + bins.half) / CUTOFF).clamp(0, bins.ext - 1).long()
            hit &= ((bins.cell[k] >= lo[w]) & (bins.cell[k] <= hi[w])).all(1)
        blocked = torch.zeros(len(pi), device=x.device).index_add_(0, w[hit], torch.ones_like(w[hit]).float())
        keep[a:a + (1 << 21)] = blocked == 0
    return i[keep], j[keep]


def _naive_delaunay(x, i, j):
    """(3-D) how many third points k have an l > k whose sphere is empty.  The finder's sphere is centred at
    x_i + c, c the circumcentre, and passes through x_i."""
    n = len(x)
    mult = torch.zeros(len(i), device=x.device, dtype=torch.float64)
    sq = x.square().sum(1)
    ids = torch.arange(n, device=x.device)
    ks, ls = torch.triu_indices(n, n, 1, device=x.device)
    for p in range(len(i)):
        a, b = int(i[p]), int(j[p])
        use = (ks != a) & (ks != b) & (ls != a) & (ls != b)
        k, l = ks[use], ls[use]
        e1, e2, e3 = (x[b] - x[a]).expand(len(k), 3), x[k] - x[a], x[l] - x[a]
        n23 = torch.linalg.cross(e2, e3)
        den = 2.0 * (e1 * n23).sum(1)
        rhs = (sq[b] - sq[a]) * n23 + (sq[k] - sq[a])[:, None] * torch.linalg.cross(e3, e1)
        centre = x[a] + (rhs + (sq[l] - sq[a])[:, None] * torch.linalg.cross(e1, e2)) / den[:, None]
        ok = den.abs() > float(np.finfo(np.float32).eps)
        k, l, centre = k[ok], l[ok], centre[ok]
        r2 = (centre - x[a]).square().sum(1)
        d2 = (centre.square().sum(1)[:, None] - 2.0 * centre @ x.T) + sq[None]
        inside = d2 <= r2[:, None]
        inside &= (ids != a) & (ids != b) & (ids != k[:, None]) & (ids != l[:, None])
        mult[p] = len(torch.unique(k[~inside.any(1)]))
    return mult


def _delaunay_2d(x, i, j):
    """Triangles on each in-cutoff edge: 2 inside the triangulation, 1 on its hull, 0 where it is not an edge."""
    mult = torch.zeros(len(i), device=x.device, dtype=torch.float64)
    step = max(1, (1 << 27) // len(x))
    inf = float("inf")
    for a in range(0, len(i), step):
        pi, pj = i[a:a + step], j[a:a + step]
        e = x[pj] - x[pi]
        m = 0.5 * (x[pi] + x[pj])
        u = x[None, :, 0] - m[:, :1]
        v = x[None, :, 1] - m[:, 1:]
        side = v * e[:, :1] - u * e[:, 1:]
        s = (u * u + v * v - 0.25 * e.square().sum(1, keepdim=True)) / (2.0 * side)
        rows = torch.arange(len(pi), device=x.device)
        left = torch.where(side > 0, s, inf)
        right = torch.where(side < 0, s, -inf)
        for t, none in ((left, inf), (right, -inf)):
            t[rows, pi] = none
            t[rows, pj] = none
        lo, hi = right.amax(1), left.amin(1)
        mult[a:a + step] = torch.where(lo <= hi, torch.isfinite(lo).double() + torch.isfinite(hi).double(), 0.0)
    return mult


def _delaunay_3d(x, i, j, around=48):
    """Distinct lesser third points over the tetrahedra on each in-cutoff edge.  Each third point k bounds the
    Voronoi face of (i, j) by a line in the bisector plane; where the other points leave a part of that line,
    its two ends are tetrahedra (i, j, k, l)."""
    n = len(x)
    once = i < j
    pi_all, pj_all = i[once], j[once]
    mult = torch.zeros(len(pi_all), device=x.device, dtype=torch.float64)
    step = max(1, (1 << 27) // (n * around))
    inf = float("inf")
    for a in range(0, len(pi_all), step):
        pi, pj = pi_all[a:a + step], pj_all[a:a + step]
        rows = torch.arange(len(pi), device=x.device)
        e = x[pj] - x[pi]
        e = e / e.norm(dim=1, keepdim=True)
        axis = torch.zeros_like(e)
        axis[rows, e.abs().argmin(1)] = 1.0
        f = torch.linalg.cross(e, axis)
        f = f / f.norm(dim=1, keepdim=True)
        g = torch.linalg.cross(e, f)
        rel = x[None] - 0.5 * (x[pi] + x[pj])[:, None]
        p, q = 2.0 * (rel @ f[:, :, None])[..., 0], 2.0 * (rel @ g[:, :, None])[..., 0]
        c = rel.square().sum(2) - 0.25 * (x[pi] - x[pj]).square().sum(1)[:, None]
        p[rows, pi], q[rows, pi], c[rows, pi] = 0.0, 0.0, 1.0
        p[rows, pj], q[rows, pj], c[rows, pj] = 0.0, 0.0, 1.0
        key = rel.square().sum(2)
        key[rows, pi], key[rows, pj] = inf, inf
        k = key.topk(min(around, n - 2), dim=1, largest=False).indices
        kp, kq, kc = p.gather(1, k), q.gather(1, k), c.gather(1, k)
        w = kp.square() + kq.square()
        # points of k's line: (base + t * direction); each other point allows a * t <= b
        bp, bq = kp * kc / w, kq * kc / w
        al = -kq[..., None] * p[:, None] + kp[..., None] * q[:, None]
        be = c[:, None] - (bp[..., None] * p[:, None] + bq[..., None] * q[:, None])
        al.scatter_(2, k[..., None], 0.0)
        be.scatter_(2, k[..., None], 1.0)
        t = be / al
        hi, hi_l = torch.where(al > 0, t, inf).min(2)
        lo, lo_l = torch.where(al < 0, t, -inf).max(2)
        some = (lo < hi) & ~((al == 0) & (be < 0)).any(2)
        big = torch.full_like(k, n)
        ends = torch.cat([torch.where(some & torch.isfinite(hi), torch.minimum(k, hi_l), big),
                          torch.where(some & torch.isfinite(lo), torch.minimum(k, lo_l), big)], 1).sort(1).values
        fresh = ends < n
        fresh[:, 1:] &= ends[:, 1:] != ends[:, :-1]
        mult[a:a + step] = fresh.sum(1).double()
    return torch.cat([pi_all, pj_all]), torch.cat([pj_all, pi_all]), torch.cat([mult, mult])


def _polarity_terms(disp, dist, pi, pj):
    """Bending (vector and angles) and alignment of the pair (i, j), each times the law's constant."""
    si, ci, sj, cj = pi[:, 0].sin(), pi[:, 0].cos(), pj[:, 0].sin(), pj[:, 0].cos()
    ti = torch.stack([si * pi[:, 1].cos(), si * pi[:, 1].sin(), ci], 1)
    tj = torch.stack([sj * pj[:, 1].cos(), sj * pj[:, 1].sin(), cj], 1)
    di, dj = (ti * disp).sum(1) / dist, (tj * disp).sum(1) / dist
    bend = -(di / dist)[:, None] * ti + (di / dist).square()[:, None] * disp
    bend = bend - (dj / dist)[:, None] * tj + (dj / dist).square()[:, None] * disp
    theta = torch.acos((disp[:, 2] / dist).clamp(-1, 1))
    turn = pi[:, 1] - torch.atan2(disp[:, 1], disp[:, 0])
    tilted = si.abs() > float(np.finfo(np.float32).eps)
    u0 = ci * theta.sin() * turn.cos() - si * theta.cos()
    u1 = torch.where(tilted, -theta.sin() * turn.sin() / si, 0.0)
    angle = pi[:, 1] - pj[:, 1]
    dot = si * sj * angle.cos() + ci * cj
    w0 = ci * sj * angle.cos() - si * cj
    w1 = torch.where(tilted, -sj * angle.sin() / si, 0.0)
    k = _f32(K_POL)
    return k * bend, k * torch.stack([dot * w0 - di * u0, dot * w1 - di * u1], 1)


def _forces(x, p, bins, finder, k_rep, k_adh):
    near = bins if bins is not None else _Bins(x, float(math.ceil(float(x.abs().max()) + 2.0)))
    i, j = near.pairs(x)
    mult = None
    if finder.endswith("gabriel"):
        i, j = _gabriel(x, bins, i, j)
    elif finder == "naive_delaunay":
        mult = _naive_delaunay(x, i, j)
    elif finder == "delaunay" and x.shape[1] == 2:
        mult = _delaunay_2d(x, i, j)
    elif finder == "delaunay":
        i, j, mult = _delaunay_3d(x, i, j)
    disp = x[i] - x[j]
    dist = disp.norm(dim=1)
    pull = _f32(k_rep) * (_f32(R_REP) - dist).clamp(min=0) - _f32(k_adh) * (dist - _f32(R_ADH)).clamp(min=0)
    f = disp * (pull / dist)[:, None]
    if mult is not None:
        f = f * mult[:, None]
    dp = None
    if p is not None:
        bend, turn = _polarity_terms(disp, dist, p[i], p[j])
        f = f + bend
        dp = torch.zeros_like(p).index_add_(0, i, turn)
    return torch.zeros_like(x).index_add_(0, i, f), dp


_MASK = (1 << 64) - 1


def _mix(z):
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _hash(step, cell, stream):
    with np.errstate(over="ignore"):
        k = cell * np.uint64(0xD1B54A32D192ED03) + np.uint64((step * 0x9E3779B97F4A7C15 +
                                                              stream * 0x94D049BB133111EB + 1) & _MASK)
        return _mix(np.uint64(SEED) ^ _mix(k)) >> np.uint64(11)


def _divide(x, step, probability):
    """Daughters a quarter of a unit from their mothers, in the order of the mothers."""
    cell = np.arange(len(x), dtype=np.uint64)
    parent = np.nonzero(_hash(step, cell, 0) <= np.uint64(math.floor(probability * 2.0**53)))[0]
    u, v = (_hash(step, cell[parent], s).astype(np.float64) / 2.0**53 for s in (1, 2))
    theta, phi = np.arccos(2.0 * u - 1.0), 2.0 * math.pi * v
    d = np.stack([np.sin(theta) * np.cos(phi), np.sin(theta) * np.sin(phi), np.cos(theta)], 1)[:, :x.shape[1]]
    mother = x[torch.from_numpy(parent).to(x.device)]
    return torch.cat([x, mother + 0.25 * torch.from_numpy(np.ascontiguousarray(d)).to(x.device)])


def _advance(x, p, half, case, k_rep=K_REP, k_adh=K_ADH):
    dt = _f32(DT)
    finder, capacity = case["finder"], _capacity(case)
    for step in range(case["steps"]):
        bins = _Bins(x, half) if finder.startswith("binned") else None

        def evaluate(y, q):
            d, dq = _forces(y, q, bins, finder, k_rep, k_adh)
            return (d - d.sum(0) / capacity if case["com"] else d), dq

        d, dq = evaluate(x, p)
        if case["integrator"] == "heun":
            d2, dq2 = evaluate(x + d * dt, None if p is None else p + dq * dt)
            d = 0.5 * (d + d2)
            dq = None if p is None else 0.5 * (dq + dq2)
        x = x + d * dt
        p = None if p is None else p + dq * dt
        if case["division"]:
            x = _divide(x, step, case["division"])
    return x, p


def exact(case, seed):
    if case["kind"] == "ensemble":
        one = dict(integrator="heun", steps=case["steps"], com=False, division=0.0)
        out = []
        for x, finder, force in _members(case, seed):
            half = float(math.ceil(float(x.abs().max()) + 2.0))
            y, _ = _advance(x.double(), None, half, dict(one, finder=finder, n=len(x)), force.k_rep, force.k_adh)
            out.append(y)
        return out
    if case["finder"] == "delaunay" and case["n"] > (45_000 if case["shape"] == "disk" else 41_000):
        return None  # over 20 seconds
    if case["finder"] == "naive_delaunay" and case["n"] > 450:
        return None
    x, p = _inputs(case, seed)
    half = float(math.ceil(float(x.abs().max()) + 2.0))
    y, q = _advance(x.double(), None if p is None else p.double(), half, case)
    return {"cells": None, "x": y, "p": q}
