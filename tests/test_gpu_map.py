"""The map pass of sparse indexes (occupancy bitmap in row order, hits queued
over units of 1 to 8 packets of 32 points) against the tree traversal, at the
sizes where a packet, a queue and a unit end and where the units grow."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 32, 33, 2_049, 60_001, 1_048_545, 2_097_121, 8_388_641]


def _device(px, py, polys):
    import torch

    return [torch.from_numpy(np.ascontiguousarray(a)).cuda()
            for a in (px, py, polys.x, polys.y, polys.ring_off, polys.part_off, polys.geom_off)]


def _sparse(n, hits):
    """Footprints in a wide frame; points uniform (sparse hits) or at footprints (every point a hit)."""
    from vibespatial_b200.testing import synthetic as syn

    polys = syn.utm_join(seed=5, n_points=16, n_polys=3_000).polys
    rng = np.random.default_rng(n)
    px = rng.uniform(polys.x.min(), polys.x.max(), n)
    py = rng.uniform(polys.y.min(), polys.y.max(), n)
    if hits == "dense":
        k = rng.integers(0, len(polys.x), n)
        px, py = polys.x[k] + rng.normal(0, 3.0, n), polys.y[k] + rng.normal(0, 3.0, n)
    px[rng.random(n) < 0.01] = np.nan
    px[rng.random(n) < 0.01] += 1e7  # outside the frame
    return px, py, polys


@pytest.mark.parametrize("hits", ["sparse", "dense"])
@pytest.mark.parametrize("n", SIZES)
def test_sparse_index_equals_tree(vsabi, ctx, n, hits):
    import torch

    px, py, polys = _sparse(n, hits)
    dev = _device(px, py, polys)
    index = vsabi.DeviceIndex(ctx, vsabi.make_polygons(*dev[2:]), learned=True)
    info = index.info()
    assert info["n_cells"] * 16 < 4 ** info["cell_level"]
    valid = torch.from_numpy((np.random.default_rng(n).random(n) > 0.05).astype(np.uint8)).cuda()
    for pts in (vsabi.make_points(*dev[:2], valid), vsabi.make_points(*dev[:2])):
        for pred in (vsabi.PRED_WITHIN, vsabi.PRED_BBOX):
            tree = index.join(pts, pred, vsabi.METHOD_RTREE)
            # (the switch changes no result and keeps few points on the grouped passes)
            cells = index.join(pts, pred, vsabi.METHOD_LEARNED, flags=vsabi.JOIN_LEARNED_NO_STAGE)
            assert torch.equal(cells[0], tree[0]) and torch.equal(cells[1], tree[1])


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("packets", [0, 2])
def test_batches_of_sparse_indexes(vsabi, ctx, mixed, packets):
    """Jobs that begin inside packets and units; with a dense index among them every job takes the other pass,
    which reads bitmaps of both orders (as it does where its packets are asked for)."""
    import torch

    from vibespatial_b200.testing import synthetic as syn

    jobs = [_sparse(n, h) for n, h in ((70_001, "sparse"), (1, "dense"), (333, "dense"), (40_010, "sparse"))]
    if mixed:
        w = syn.star_join(seed=2, n_points=20_003, n_polys=400)
        jobs.insert(2, (w.px, w.py, w.polys))
    dev = [_device(*j) for j in jobs]
    indexes = [vsabi.DeviceIndex(ctx, vsabi.make_polygons(*d[2:]), learned=True) for d in dev]
    start = np.concatenate([[0], np.cumsum([len(j[0]) for j in jobs])]).astype(np.int64)
    px, py = torch.cat([d[0] for d in dev]), torch.cat([d[1] for d in dev])
    plan = vsabi.BatchPlan(ctx, indexes, vsabi.make_points(px, py), start,
                           options={"method": vsabi.METHOD_LEARNED, "learned_map_packets": packets})
    left, right, _ = plan.run(vsabi.PRED_WITHIN)
    got = set(zip(left.tolist(), right.tolist()))
    want = set()
    for s, d, index in zip(start, dev, indexes):
        one = index.join(vsabi.make_points(*d[:2]), vsabi.PRED_WITHIN, vsabi.METHOD_RTREE)
        want |= set(zip((one[0] + int(s)).tolist(), one[1].tolist()))
    assert got == want and len(got) == left.numel()


def _map_kernels(run):
    """Names of the map kernels that a call launches."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    run()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        run()
        torch.cuda.synchronize()
    return {n for e in prof.events() for n in ("learned_map_sparse_kernel", "learned_map_kernel") if n in e.name}


@pytest.mark.parametrize("hits", ["sparse", "dense"])
@pytest.mark.parametrize("n", [2**21 - 1, 2**21, 2**21 + 33, 2**22 + 127, 2**23 - 1, 2**23 + 257])
def test_where_the_sparse_pass_begins(vsabi, ctx, n, hits):
    """The sizes where the pass and its units change, with the last unit, packet and lane full and cut off."""
    import torch

    px, py, polys = _sparse(n, hits)
    dev = _device(px, py, polys)
    index = vsabi.DeviceIndex(ctx, vsabi.make_polygons(*dev[2:]), learned=True)
    pts = vsabi.make_points(*dev[:2])
    tree = index.join(pts, vsabi.PRED_WITHIN, vsabi.METHOD_RTREE)
    cells = index.join(pts, vsabi.PRED_WITHIN, vsabi.METHOD_LEARNED)
    assert torch.equal(cells[0], tree[0]) and torch.equal(cells[1], tree[1])


def test_every_launch_shape_takes_the_sparse_pass(vsabi, ctx):
    """A plan with any launch shape (tuned, from the cache, or none) maps the points of sparse indexes by their own
    pass from 2^21 points on, as a join does, and by the other below; jobs begin inside units and packets."""
    import torch

    jobs = [_sparse(n, h) for n, h in ((2**21 - 7, "sparse"), (1, "dense"), (333, "dense"), (70_001, "sparse"))]
    dev = [_device(*j) for j in jobs]
    indexes = [vsabi.DeviceIndex(ctx, vsabi.make_polygons(*d[2:]), learned=True) for d in dev]
    start = np.concatenate([[0], np.cumsum([len(j[0]) for j in jobs])]).astype(np.int64)
    px, py = torch.cat([d[0] for d in dev]), torch.cat([d[1] for d in dev])
    want = []
    for s, d, index in zip(start, dev, indexes):
        one = index.join(vsabi.make_points(*d[:2]), vsabi.PRED_WITHIN, vsabi.METHOD_RTREE)
        want.append((one[0].to(torch.int64) + int(s)) * 2**20 + one[1])
    want = torch.cat(want).sort()[0]
    pts = vsabi.make_points(px, py)
    few = vsabi.make_points(px[:-70_001 - 334], py[:-70_001 - 334])
    for shape in ({}, {"learned_map_packets": 1}, {"learned_map_packets": 2, "learned_map_blocks_per_sm": 2}):
        options = dict(shape, method=vsabi.METHOD_LEARNED)
        plan = vsabi.BatchPlan(ctx, indexes, pts, start, options=options)
        left, right, _ = plan.run(vsabi.PRED_WITHIN)
        assert torch.equal((left.to(torch.int64) * 2**20 + right).sort()[0], want)
        assert _map_kernels(lambda: plan.run(vsabi.PRED_WITHIN)) == {"learned_map_sparse_kernel"}
        plan.close()
        plan = vsabi.BatchPlan(ctx, indexes[:1], few, start[:2], options=options)
        assert _map_kernels(lambda: plan.run(vsabi.PRED_WITHIN)) == {"learned_map_kernel"}
        plan.close()
