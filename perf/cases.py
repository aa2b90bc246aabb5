"""Performance cases of the periodic Delaunay library: the calls that its users make, through the
public Python classes (`DelaunayGPU`, `DelaunayBatch`, `MDGraph`), over the range of sizes and
options that they make them with.

- `build`: one `globalDelaunayTriangulation` of positions already on the GPU, safety mode on
  (the default), into arrays that the program keeps.
- `repair`: one `testAndRepairDelaunayTriangulation` with the next frame of a trajectory, the
  arrays holding the triangulation of the previous one.  A state holds two frames, sigma apart
  per axis, and its passes go from one to the other and back.
- `md`: one replay of a captured graph of MD steps (displacement and repair on the device).

Point sets: `uniform` (unit density), `lattice` (jittered triangular lattice, rectangular
box), `square` (the reference driver's square lattice, each site up to a quarter spacing off),
`mixture` (64 Gaussian clusters, large density contrast).  `hex` puts uniform points into a
60-degree general box.  `sets` > 1 is an ensemble of independent sets with log-uniform sizes.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from gpudelaunaytriangulation_b200.delaunay import DelaunayBatch, DelaunayGPU, PeriodicBox

# what a case may leave out
DEFAULTS = {
    "points": "uniform", "n": 0, "cell": 1.0, "stride": 20, "fp64": False, "hex": False,
    "sets": 1, "lo": 0, "hi": 0, "sizes_seed": 7, "sigma": 0.0, "steps": 0,
    "budget": -1, "shape": -1, "pieces": 1,
}


def listed():
    return [
        # A triangulation of a small cell or particle model: launches and latency only.
        {"name": "build_1k", "kind": "build", "n": 1000, "stride": 16},
        # The reference driver's order of magnitude (and the golden fixture's size).
        {"name": "build_10k", "kind": "build", "n": 10_000, "stride": 16},
        # An ordinary simulation, an odd size, cells a little over the mean spacing.
        {"name": "build_130k", "kind": "build", "n": 131_071, "cell": 1.2, "stride": 16},
        # The caller asks for float64 predicates.
        {"name": "build_1m_fp64", "kind": "build", "n": 1_000_000, "fp64": True},
        # The headline benchmark's triangulation.
        {"name": "build_4m", "kind": "build", "n": 4_194_304},
        # A crystal: near-cocircular neighbours, a rectangular box.
        {"name": "build_lattice_1m", "kind": "build", "points": "lattice", "n": 1_000_000, "stride": 16},
        # Strongly clustered points, with the settings that the autotuner picked for them.
        {"name": "build_mixture_1m", "kind": "build", "points": "mixture", "n": 1_000_000, "stride": 32,
         "cell": 0.18, "budget": 512, "shape": 4, "pieces": 4},
        # A sheared simulation cell: the general-box kernels.
        {"name": "build_hex_1m", "kind": "build", "n": 1_000_003, "hex": True},
        # One MD frame of a small system: a handful of edges change.
        {"name": "repair_10k", "kind": "repair", "n": 10_000, "sigma": 0.02, "stride": 16},
        # One frame with large moves (many flips, some inverted fans), an odd size.
        {"name": "repair_1m", "kind": "repair", "n": 999_983, "sigma": 0.05},
        # The headline benchmark's repair.
        {"name": "repair_4m", "kind": "repair", "n": 4_194_304, "sigma": 0.02},
        # MD steps of an ensemble of independent systems, replayed from a graph.
        {"name": "md_ensemble", "kind": "md", "sets": 256, "lo": 1000, "hi": 65_536, "sigma": 0.01, "steps": 5},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["build", "build", "build", "build", "repair", "repair", "repair", "md"])
    if what == "md":
        # between one system and an ensemble
        sets = _log_uniform(rng, 1, 256)
        return {"kind": "md", "sets": sets, "lo": 1000, "hi": 65_536, "sizes_seed": rng.randrange(1, 1 << 20),
                "sigma": round(rng.uniform(0.004, 0.02), 4), "steps": rng.randint(1, 5)}
    if what == "repair":
        c = {"kind": "repair", "n": _log_uniform(rng, 1000, 4_000_000), "sigma": round(rng.uniform(0.005, 0.06), 4)}
        c["hex"] = rng.random() < 0.2
        c["fp64"] = rng.random() < 0.2
        c["cell"] = round(rng.uniform(0.85, 1.3), 3)
        return c
    points = rng.choice(["uniform", "uniform", "uniform", "lattice", "square", "mixture", "ensemble"])
    if points == "ensemble":
        return {"kind": "build", "sets": _log_uniform(rng, 2, 200), "lo": 1000, "hi": 65_536,
                "sizes_seed": rng.randrange(1, 1 << 20), "cell": round(rng.uniform(0.85, 1.3), 3)}
    if points == "mixture":
        return {"kind": "build", "points": "mixture", "n": _log_uniform(rng, 200_000, 1_000_000), "stride": 32,
                "cell": 0.18, "budget": 512, "shape": 4, "pieces": rng.randint(1, 4)}
    c = {"kind": "build", "points": points, "n": _log_uniform(rng, 500, 4_000_000)}
    c["cell"] = round(rng.uniform(0.85, 1.3), 3)
    c["fp64"] = rng.random() < 0.2 and c["n"] < 2_000_000
    c["hex"] = points == "uniform" and rng.random() < 0.2
    return c


def _full(case):
    return {**DEFAULTS, **case}


def _sizes(c):
    u = np.random.RandomState(c["sizes_seed"]).random_sample(c["sets"])
    return np.floor(np.exp(math.log(c["lo"]) + u * (math.log(c["hi"]) - math.log(c["lo"])))).astype(np.int64)


def _lattice_grid(n):
    """Rows and columns of the triangular lattice nearest to n sites (an even number of rows)."""
    ny = max(2, 2 * int(round(math.sqrt(n) / 2)))
    return max(2, int(round(n / ny))), ny


def _count(c):
    if c["sets"] > 1 or c["kind"] == "md":
        return int(_sizes(c).sum())
    if c["points"] == "lattice":
        nx, ny = _lattice_grid(c["n"])
        return nx * ny
    return c["n"]


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _points(c, g):
    """(points, box) of a single set, the mean spacing near one."""
    n = c["n"]
    if c["points"] == "lattice":
        nx, ny = _lattice_grid(n)
        h = math.sqrt(3.0) / 2.0
        j, i = torch.meshgrid(torch.arange(ny, device="cuda", dtype=torch.float64),
                              torch.arange(nx, device="cuda", dtype=torch.float64), indexing="ij")
        p = torch.stack([(i + 0.5 * torch.remainder(j, 2.0)).reshape(-1), (j * h).reshape(-1)], dim=1)
        p = p + (2.0 * _rand(g, nx * ny, 2) - 1.0) * 1e-4
        # the sites are numbered from one of their own: on a lattice nothing else tells two sets apart
        p = torch.roll(p, int(_rand(g, 1).item() * nx * ny), dims=0)
        box = PeriodicBox(float(nx), ny * h)
        return box.putInBoxReal(p), box
    L = math.sqrt(n)
    box = PeriodicBox(L, L)
    if c["points"] == "square":
        k = int(math.ceil(L))
        site = torch.arange(n, device="cuda")
        p = torch.stack([torch.div(site, k, rounding_mode="floor"), site % k], dim=1).double() + 0.5
        p = (p + (2.0 * _rand(g, n, 2) - 1.0) * 0.25) * (L / k)
        return box.putInBoxReal(p), box
    if c["points"] == "mixture":
        L *= 1.024
        box = PeriodicBox(L, L)
        centres = _rand(g, 64, 2) * L
        which = torch.floor(_rand(g, n) * 64).long()
        return box.putInBoxReal(centres[which] + 2.0 * _randn(g, n, 2)), box
    u = _rand(g, n, 2)
    if c["hex"]:
        a = math.sqrt(n / (math.sqrt(3.0) / 2.0))
        box = PeriodicBox.general(a, 0.5 * a, 0.0, a * math.sqrt(3.0) / 2.0)
        m = torch.tensor([[box.Lx, box.xy], [box.yx, box.Ly]], device="cuda", dtype=torch.float64)
        return (u @ m.T).contiguous(), box
    return u * L, box


def _md_start(c, seed):
    """(points, sizes, box sides) of an ensemble of uniform sets at unit density."""
    sizes = _sizes(c)
    side = np.sqrt(sizes.astype(np.float64))
    scale = torch.from_numpy(np.repeat(side, sizes)).cuda()
    return _rand(_generator(seed), int(sizes.sum()), 2) * scale[:, None], sizes, side


def prepare(case, seed):
    c = _full(case)
    g = _generator(seed)
    stride = c["stride"]
    if c["sets"] > 1 or c["kind"] == "md":
        p, sizes, side = _md_start(c, seed)
        d = DelaunayBatch(sizes.tolist(), [(float(s), float(s)) for s in side], stride, c["cell"])
    else:
        p, box = _points(c, g)
        d = DelaunayGPU(len(p), stride, c["cell"], box)
    if c["fp64"]:
        d.setPrecision(False)
    if c["budget"] >= 0:
        d.setWorkBudget(c["budget"])
    if c["shape"] >= 0:
        d.setKernelShape(c["shape"])
    if c["pieces"] > 1:
        d.setDeferredOverlap(c["pieces"])
    n = len(p)
    s = {"kind": c["kind"], "d": d, "p": p, "tri": torch.zeros(stride * n, dtype=torch.int32, device="cuda"),
         "nn": torch.zeros(n, dtype=torch.int32, device="cuda")}
    if c["kind"] == "build":
        return s
    # a running simulation: the triangulation of the present positions is there
    d.globalDelaunayTriangulation(p, s["tri"], s["nn"])
    s["column"] = torch.arange(stride, dtype=torch.int32, device="cuda")
    if c["kind"] == "repair":
        q = p + c["sigma"] * _randn(g, n, 2)
        s["frames"] = [p, d.Box.putInBoxReal(q)]
        s["at"] = 0
        return s
    s["stream"] = torch.cuda.Stream()
    s["stream"].wait_stream(torch.cuda.current_stream())
    s["graph"] = d.mdGraph(p, s["tri"], s["nn"], c["sigma"], seed=int(seed) + 1, steps=c["steps"], rounds=4,
                           stream=s["stream"])
    return s


def _padded(s):
    """Rows as padded arrays: what a repair leaves past a ring's length is not specified, so a
    program that hands whole rows on blanks it."""
    rows = s["tri"].view(len(s["nn"]), -1)
    rows.masked_fill_(s["column"] >= s["nn"][:, None], -1)
    return rows


def run(s):
    d = s["d"]
    if s["kind"] == "build":
        return d.globalDelaunayTriangulation(s["p"], s["tri"], s["nn"])
    if s["kind"] == "repair":
        s["at"] ^= 1
        d.testAndRepairDelaunayTriangulation(s["frames"][s["at"]], s["tri"], s["nn"])
        return _padded(s), s["nn"]
    with torch.cuda.stream(s["stream"]):
        s["graph"].launch(s["stream"])
        return s["p"], _padded(s), s["nn"]


def work(case):
    """Compulsory traffic: every position read (16 B), a ring of six neighbours (24 B) and its
    length (4 B) per point, written by a build, read by a repair; an MD step also writes the
    position.  The arithmetic is not counted: it is decisions, and how many a method takes is
    the method's own."""
    c = _full(case)
    n = _count(c)
    if c["kind"] == "md":
        return {"bytes": 60.0 * n * c["steps"], "flops": 0.0}
    return {"bytes": 44.0 * n, "flops": 0.0}


_U64 = (1 << 64) - 1


def _splitmix(z):
    z = z + np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def exact(case, seed):
    """The MD steps' positions: normals of (seed, step, point) by Box-Muller, wrapped into each
    set's box.  Rings are whole numbers and have no value of their own here."""
    c = _full(case)
    if c["kind"] != "md":
        return None
    p, sizes, side = _md_start(c, seed)
    p = p.cpu().numpy()
    box = np.repeat(side, sizes)[:, None]
    i = np.arange(len(p), dtype=np.uint64)
    key = np.uint64((int(seed) + 1) & _U64)
    with np.errstate(over="ignore"):
        for step in range(c["steps"]):
            h = _splitmix(key ^ _splitmix(np.uint64((step * 0x100000001B3) & _U64) + i))
            h2 = _splitmix(h)
            r = c["sigma"] * np.sqrt(-2.0 * np.log(((h >> np.uint64(11)) + np.uint64(1)) / 9007199254740993.0))
            t = 2.0 * math.pi * ((h2 >> np.uint64(11)) / 9007199254740992.0)
            p = p + r[:, None] * np.stack([np.cos(t), np.sin(t)], axis=1)
            p = np.where(p >= box, p - box, np.where(p < 0.0, p + box, p))
            p[p >= box] = 0.0
    return [p, None, None]
