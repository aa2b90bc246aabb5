"""The first stage of builds and rebuilds (k_star) against the incremental kernels: a work
budget below its scans leaves every point to them, and both must give the same arrays, for
every form of input the first stage accepts (windows of every size, box edges, ragged and tiny
sets, dense and sparse cells, both precisions, general boxes, batches, kept cell lists)."""
import numpy as np
import pytest

from gpudelaunaytriangulation_b200 import workloads as W

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

HEX = (1.0, 0.5, 0.0, np.sqrt(3.0) / 2.0)


def _rings(pts, box, cell, incremental, fp64=False, sizes=None, moved=None, stride=24, check=False):
    from gpudelaunaytriangulation_b200.delaunay import DelaunayBatch, DelaunayGPU

    d = DelaunayBatch(sizes, box, stride, cell) if sizes is not None else DelaunayGPU(len(pts), stride, cell, box)
    d.setPrecision(not fp64)
    d.setCheckMode(check)
    if incremental:
        d.setWorkBudget(255)
    P = torch.from_numpy(pts).cuda()
    tri, nn = d.globalDelaunayTriangulation(P)
    st = d.stats()
    assert st["mismatches"] == 0 and st["error_flags"] & ~32 == 0, st
    if moved is not None:
        d.setFlipRepair(False)   # every flagged point through the rebuild rounds
        P.copy_(torch.from_numpy(moved))
        tri.view(len(pts), -1).masked_fill_(torch.arange(stride, device="cuda") >= nn[:, None], 0)
        d.testAndRepairDelaunayTriangulation(P, tri, nn)
        assert d.stats()["error_flags"] & ~32 == 0
        tri.view(len(pts), -1).masked_fill_(torch.arange(stride, device="cuda") >= nn[:, None], 0)
    return tri, nn


def _same(*args, **kw):
    b = _rings(*args, True, **kw)
    for check in (False, True):   # (check mode: every decision contradicted by float64 is counted)
        a = _rings(*args, False, check=check, **kw)
        assert torch.equal(a[1], b[1])
        assert torch.equal(a[0], b[0])


@pytest.mark.parametrize("n", [24, 63, 64, 65, 700, 19_999, 20_001, 150_000])
@pytest.mark.parametrize("cell", [0.45, 0.8, 1.0, 1.3, 1.7, 2.6])
def test_uniform_sets(n, cell):
    L = float(np.sqrt(n))
    _same(W.uniform_points(n, L, 500 + n), (L, L), cell)


@pytest.mark.parametrize("aspect", [0.04, 0.3, 5.0])
def test_rectangles(aspect):
    n = 30_000
    Lx, Ly = float(np.sqrt(n * aspect)), float(np.sqrt(n / aspect))
    _same(W.uniform_points(n, Lx, 77, Ly), (Lx, Ly), 1.0)


@pytest.mark.parametrize("jitter", [1e-7, 1e-4, 0.05])
def test_lattices(jitter):
    # collinear candidates at every angle, near-cocircular ones on every circle
    pts, Lx, Ly = W.triangular_lattice(150, 150, jitter=jitter, seed=8)
    _same(pts, (Lx, Ly), 1.0)


@pytest.mark.parametrize("cell", [0.2, 0.5, 1.0])
def test_clusters(cell):
    pts, L = W.gaussian_mixture(60_000, components=12, sigma=3.0, L=260.0, seed=6)
    _same(pts, (L, L), cell)


@pytest.mark.parametrize("scale", [1e-9, 1e9])
def test_float64_and_units(scale):
    # the same set in other units: far from one, squares leave the filter's range
    n = 25_000
    L = float(np.sqrt(n))
    pts = W.uniform_points(n, L, 91)
    for fp64 in (False, True):
        _same(pts, (L, L), 1.0, fp64=fp64)
        _same(pts * scale, (L * scale, L * scale), scale, fp64=fp64)


def test_general_box():
    n = 25_000
    s = float(np.sqrt(n / (np.sqrt(3.0) / 2.0)))
    u = W.uniform_points(n, 1.0, 92)
    m = np.array(HEX).reshape(2, 2) * s
    for shift in (0.0, 3.0):   # outside the primary cell too
        pts = np.ascontiguousarray((u + np.floor(shift * W.uniform_points(n, 1.0, 93))) @ m.T)
        for fp64 in (False, True):
            _same(pts, tuple(m.reshape(-1)), 1.0, fp64=fp64)


def test_batch():
    sizes = np.array([30, 5000, 0, 64, 40_000, 1000], dtype=np.int64)
    boxes = np.stack([np.sqrt(np.maximum(sizes, 1).astype(np.float64))] * 2, axis=1)
    pts = np.concatenate([W.uniform_points(int(k), float(L), 600 + i)
                          for i, (k, L) in enumerate(zip(sizes, boxes[:, 0])) if k > 0])
    _same(pts, boxes, 1.0, sizes=sizes)


@pytest.mark.parametrize("sigma", [0.05, 0.3])
@pytest.mark.parametrize("n", [900, 60_000])
def test_rebuild_rounds(n, sigma):
    # cell lists older than the positions, points across the box's edge among them
    L = float(np.sqrt(n))
    pts = W.uniform_points(n, L, 95)
    _same(pts, (L, L), 1.0, moved=W.displace(pts, sigma, L, L, 96))


@pytest.mark.parametrize("n", [4095, 4096, 4097, 16_384, 16_385])
def test_small_set_kernels(n):
    # the one-block binning and flips on either side of the sizes they are taken for: the same
    # cell order and triangulations as the launches of a large set (a batch with an empty
    # large set beside it goes the other way)
    from gpudelaunaytriangulation_b200.delaunay import DelaunayBatch, DelaunayGPU

    L = float(np.sqrt(n))
    pts = W.uniform_points(n, L, 700 + n)
    moved = W.displace(pts, 0.05, L, L, 701)
    big = W.uniform_points(20_000, 200.0, 702)
    one = DelaunayGPU(n, 20, 1.0, (L, L))
    two = DelaunayBatch([n, 20_000], [(L, L), (200.0, 200.0)], 20, 1.0)
    P1 = torch.from_numpy(pts).cuda()
    P2 = torch.from_numpy(np.concatenate([pts, big])).cuda()
    t1, k1 = one.globalDelaunayTriangulation(P1)
    t2, k2 = two.globalDelaunayTriangulation(P2)
    assert torch.equal(k1, k2[:n]) and torch.equal(t1, t2[: t1.numel()])
    assert torch.equal(one.cellOrder(), two.cellOrder()[:n])
    P1.copy_(torch.from_numpy(moved))
    P2[:n].copy_(P1)
    one.testAndRepairDelaunayTriangulation(P1, t1, k1)
    two.testAndRepairDelaunayTriangulation(P2, t2, k2)
    rows = torch.arange(20, device="cuda")[None, :] < k1[:, None]
    assert torch.equal(k1, k2[:n]) and torch.equal(t1.view(n, -1)[rows], t2[: t1.numel()].view(n, -1)[rows])
    assert one.validate(P1, t1, k1)["valid"] == 1
    assert one.stats()["flips"] > 0


# Sets of more than 12,000 points, which k_star takes (up to that many k_wrap takes a build whole), of
# more than 48,000 in two passes.
BIG = 50_000


def _build_big(pts, box, cell, incremental, fp64=False, sizes=None, moved=None, stride=24, check=False):
    from gpudelaunaytriangulation_b200.delaunay import DelaunayBatch, DelaunayGPU

    d = DelaunayBatch(sizes, box, stride, cell) if sizes is not None else DelaunayGPU(len(pts), stride, cell, box)
    d.setPrecision(not fp64)
    d.setCheckMode(check)
    if incremental:
        d.setWorkBudget(255)
    P = torch.from_numpy(pts).cuda()
    tri, nn = d.globalDelaunayTriangulation(P)
    st = d.stats()
    assert st["mismatches"] == 0 and st["error_flags"] & ~32 == 0, st
    if moved is not None:
        d.setFlipRepair(False)   # every flagged point through the rebuild rounds
        P.copy_(torch.from_numpy(moved))
        d.testAndRepairDelaunayTriangulation(P, tri, nn)
        again = d.stats()
        assert again["mismatches"] == 0 and again["error_flags"] & ~32 == 0, again
        assert again["flagged"] > 20_000   # the first round's list is k_star's
        tri.view(len(pts), -1).masked_fill_(torch.arange(stride, device="cuda") >= nn[:, None], 0)
    return tri, nn, st


def _same_big(*args, **kw):
    b = _build_big(*args, True, **kw)
    for check in (False, True):
        a = _build_big(*args, False, check=check, **kw)
        # the incremental path builds in one launch, the first stage in one or two of k_star and k_wrap
        assert a[2]["launches"] == b[2]["launches"] + (2 if len(args[0]) > 48_000 else 1)
        assert torch.equal(a[1], b[1])
        assert torch.equal(a[0], b[0])


def _uneven_points(n, part, spread, seed):
    """`part` of n points in one row of unit cells, over its whole length or (spread) normal about
    its middle, the others uniform; returns (points, L)."""
    L = float(np.sqrt(n))
    k = int(part * n)
    h = L / int(L)
    pts = W.uniform_points(n, L, seed)
    pts[:k, 1] = (int(L / 2) + pts[:k, 1] / L) * h
    if spread:
        pts[:k, 0] = L / 2 + spread * W.normal_pairs(seed + 1, k)[:, 0]
    return W.wrap(pts, L, L), L


@pytest.mark.parametrize("n,part,spread", [(60_000, 0.56, 0.0), (60_000, 0.7, 0.0), (100_000, 0.7, 0.0),
                                           (64_000, 0.5625, 6.0)])
def test_most_points_in_one_row_of_cells(n, part, spread):
    # neighbouring rows lie more than half the set and more than 32,767 slots apart in the cell
    # order, in windows that do not cross the box's edge: slots as 16-bit offsets
    pts, L = _uneven_points(n, part, spread, 1)
    _same_big(pts, (L, L), 1.0, stride=64)


@pytest.mark.parametrize("n", [12_001, 40_001, 48_000, 48_001, 131_071])
@pytest.mark.parametrize("cell", [0.45, 0.8, 1.0, 1.7, 2.6])
def test_big_uniform_sets(n, cell):
    L = float(np.sqrt(n))
    _same_big(W.uniform_points(n, L, 510 + n), (L, L), cell)


@pytest.mark.parametrize("aspect", [0.005, 0.04, 0.3, 5.0])
def test_big_rectangles(aspect):
    Lx, Ly = float(np.sqrt(BIG * aspect)), float(np.sqrt(BIG / aspect))
    _same_big(W.uniform_points(BIG, Lx, 78, Ly), (Lx, Ly), 1.0)


@pytest.mark.parametrize("jitter", [1e-7, 1e-4, 0.05])
def test_big_lattices(jitter):
    # collinear candidates at every angle (triangular), four near-cocircular ones round every
    # square
    pts, Lx, Ly = W.triangular_lattice(222, 222, jitter=jitter, seed=8)
    _same_big(pts, (Lx, Ly), 1.0)
    pts, L = W.square_lattice(222 * 222, phase=jitter, seed=8)
    _same_big(pts, (L, L), 1.0)


@pytest.mark.parametrize("cell", [0.2, 1.0])
def test_big_clusters(cell):
    pts, L = W.gaussian_mixture(60_000, components=12, sigma=3.0, L=260.0, seed=6)
    for fp64 in (False, True):
        _same_big(pts, (L, L), cell, fp64=fp64, stride=32)


@pytest.mark.parametrize("scale", [1e-9, 1.0, 1e9])
@pytest.mark.parametrize("fp64", [False, True])
def test_big_float64_and_units(scale, fp64):
    L = float(np.sqrt(BIG))
    pts = W.uniform_points(BIG, L, 191)
    _same_big(pts * scale, (L * scale, L * scale), scale, fp64=fp64)


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("shift", [0.0, 3.0])
def test_big_general_box(fp64, shift):
    m = np.array(HEX).reshape(2, 2) * float(np.sqrt(BIG / (np.sqrt(3.0) / 2.0)))
    u = W.uniform_points(BIG, 1.0, 192)
    # (shift: outside the primary cell too)
    pts = np.ascontiguousarray((u + np.floor(shift * W.uniform_points(BIG, 1.0, 193))) @ m.T)
    _same_big(pts, tuple(m.reshape(-1)), 1.0, fp64=fp64)


def test_big_batch():
    sizes = np.array([5000, 0, 64, 50_000, 1000, 300], dtype=np.int64)
    boxes = np.stack([np.sqrt(np.maximum(sizes, 1).astype(np.float64))] * 2, axis=1)
    pts = np.concatenate([W.uniform_points(int(k), float(L), 650 + i)
                          for i, (k, L) in enumerate(zip(sizes, boxes[:, 0])) if k > 0])
    for fp64 in (False, True):
        _same_big(pts, boxes, 1.0, sizes=sizes, fp64=fp64)


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("sigma", [0.1, 0.3])
@pytest.mark.parametrize("n", [46_000, 90_000])
def test_big_rebuild_rounds(n, fp64, sigma):
    # lists of more than 20,000 points (one pass) and 48,000 (both), with kept (0.1) and new cell lists
    L = float(np.sqrt(n))
    pts = W.uniform_points(n, L, 195)
    _same_big(pts, (L, L), 1.0, moved=W.displace(pts, sigma, L, L, 196), fp64=fp64)
    m = np.array(HEX).reshape(2, 2) * float(np.sqrt(n / (np.sqrt(3.0) / 2.0)))
    pts = np.ascontiguousarray(W.uniform_points(n, 1.0, 197) @ m.T)
    _same_big(pts, tuple(m.reshape(-1)), 1.0, moved=pts + sigma * W.normal_pairs(198, n), fp64=fp64)


def _strips(width, sizes, seed):
    boxes = np.stack([np.full(len(sizes), width), sizes / width], axis=1)
    return np.concatenate([W.uniform_points(int(k), width, seed + i, float(b[1]))
                           for i, (k, b) in enumerate(zip(sizes, boxes))]), boxes


@pytest.mark.parametrize("rebuild", [False, True])
@pytest.mark.parametrize("width", [4.7, 5.2, 6.2])
@pytest.mark.parametrize("cell", [0.3, 0.45, 0.6, 0.8, 1.0])
@pytest.mark.parametrize("big", [8_000, 60_000])
def test_narrow_boxes(big, cell, width, rebuild):
    # circles close to half the box and past it (where circles pass half the box, flag 32, the
    # nearest images still give one answer): windows over the whole short axis.  Beside a large set,
    # so that the hull kernels are taken, of up to 12,000 points and more
    sizes = np.arange(60, 150, 3)
    pts, boxes = _strips(width, sizes, 800)
    L = float(np.sqrt(big))
    pts = np.concatenate([pts, W.uniform_points(big, L, 802)])
    sizes = np.append(sizes, big)
    boxes = np.concatenate([boxes, [[L, L]]])
    moved = None
    if rebuild:
        every = np.repeat(boxes, sizes, axis=0)
        moved = np.mod(pts + 0.2 * W.normal_pairs(801, len(pts)), every)
        moved = np.where(moved >= every, 0.0, moved)
    b = _rings(pts, boxes, cell, True, sizes=sizes, moved=moved)
    for fp64 in (False, True):
        a = _rings(pts, boxes, cell, False, sizes=sizes, moved=moved, fp64=fp64)
        assert torch.equal(a[1], b[1])
        assert torch.equal(a[0], b[0])


@pytest.mark.parametrize("width,sizes", [(2.5, [12_000]), (4.2, [3_000]), (4.2, [60_000]), (5.2, [100_000]),
                                         (4.0, [16] * 2500), (5.0, [25] * 1600)])
def test_mostly_narrow_boxes(width, sizes):
    # sets whose circles pass half the box by the thousand: a thread per point, not a warp each
    from gpudelaunaytriangulation_b200.delaunay import DelaunayBatch

    sizes = np.array(sizes)
    if len(sizes) == 1:
        pts, boxes = _strips(width, sizes, 810)
    else:
        pts = np.concatenate([W.square_lattice(int(k), 0.25, 810 + i)[0] for i, k in enumerate(sizes)])
        boxes = np.full((len(sizes), 2), width)
    d = DelaunayBatch(sizes, boxes, 24, 1.0)
    d.globalDelaunayTriangulation(torch.from_numpy(pts).cuda())
    assert d.stats()["exact_points"] < len(pts) // 100
    a, b = (_rings(pts, boxes, 1.0, inc, sizes=sizes) for inc in (False, True))
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])


@pytest.mark.parametrize("pieces", [1, 2, 8])
def test_pieces_of_a_large_build(pieces):
    # a build of 100,000 points in pieces (12,500 points each in 8): every piece in two launches of
    # k_star and one of k_wrap, and the rings of the whole
    from gpudelaunaytriangulation_b200.delaunay import DelaunayGPU

    n = 100_000
    L = float(np.sqrt(n))
    P = torch.from_numpy(W.uniform_points(n, L, 95)).cuda()
    out, launches = [], []
    for budget in (1024, 255):
        d = DelaunayGPU(n, 24, 1.0, (L, L))
        d.setDeferredOverlap(pieces)
        d.setWorkBudget(budget)
        out.append(d.globalDelaunayTriangulation(P))
        launches.append(d.stats()["launches"])
    assert launches[0] == launches[1] + 2 * pieces
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("n", [13_225, 62_500])
@pytest.mark.parametrize("jitter", [1e-3, 1e-6, 1e-9])
def test_near_cocircular_squares(jitter, n, fp64):
    # the four corners of every square within rounding of a circle: the diagonals that are no edges
    # are taken out of the ring by the float64 decision, in the first pass (25 candidates a point; a
    # second kernel would scan as many again)
    from gpudelaunaytriangulation_b200.delaunay import DelaunayGPU

    pts, L = W.square_lattice(n, phase=jitter, seed=5)
    d = DelaunayGPU(n, 16, 1.0, (L, L))
    d.setPrecision(not fp64)
    d.globalDelaunayTriangulation(torch.from_numpy(pts).cuda())
    st = d.stats()
    assert st["candidates"] <= 26 * n and st["exact_points"] <= n // 1000, st
    _same_big(pts, (L, L), 1.0, fp64=fp64)


@pytest.mark.parametrize("n", [1000, 10_000, 10_001, 16_384])
@pytest.mark.parametrize("sigma", [0.02, 0.15])
@pytest.mark.parametrize("general", [False, True])
def test_flip_rounds_of_small_sets(general, sigma, n):
    # all flip rounds in one block or one cluster (long lists at the larger sigma), five moves in a
    # row: the rings of a fresh build
    from gpudelaunaytriangulation_b200.delaunay import DelaunayGPU

    L = float(np.sqrt(n))
    m = np.array(HEX).reshape(2, 2) * float(np.sqrt(n / (np.sqrt(3.0) / 2.0)))
    box = tuple(m.reshape(-1)) if general else (L, L)
    pts = W.uniform_points(n, 1.0, 720 + n) @ m.T if general else W.uniform_points(n, L, 720 + n)
    d = DelaunayGPU(n, 24, 1.0, box)
    P = torch.from_numpy(np.ascontiguousarray(pts)).cuda()
    tri, nn = d.globalDelaunayTriangulation(P)
    flips = 0
    for step in range(5):
        pts = pts + sigma * W.normal_pairs(721 + step, n)
        if not general:
            pts = W.wrap(pts, L, L)
        P.copy_(torch.from_numpy(pts))
        d.testAndRepairDelaunayTriangulation(P, tri, nn)
        flips += d.stats()["flips"]
        assert d.stats()["error_flags"] == 0
        fresh, k = DelaunayGPU(n, 24, 1.0, box).globalDelaunayTriangulation(P)
        assert torch.equal(nn, k)
        rows = torch.arange(24, device="cuda")[None, :] < k[:, None]
        # (a repaired row may begin at another of its entries)
        a, b = (torch.where(rows, t.view(n, -1), -1).sort(dim=1).values for t in (tri, fresh))
        assert torch.equal(a, b)
        assert d.validate(P, tri, nn)["valid"] == 1
    assert flips > 0
