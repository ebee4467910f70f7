"""The direct learned join (few points, one launch) against the grouped one.

An ablation switch that changes no result (records read without staging) keeps
a call on the grouped passes, so both answer the same inputs here.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 32, 33, 255, 257, 5_000, 40_000]


def _inputs(kind, n):
    from vibespatial_b200.testing import synthetic as syn

    w = {"star": lambda: syn.star_join(seed=n, n_points=n, n_polys=900),
         "zipf": lambda: syn.zipf_join(seed=n, n_points=n, n_polys=4_000, sites=8),
         "degenerate": lambda: syn.degenerate_join(seed=n, n_points=max(n, 10), n_polys=150, extent=1024.0)}[kind]()
    px, py = w.px[:n].copy(), w.py[:n].copy()
    rng = np.random.default_rng(n)
    valid = (rng.random(n) > 0.05).astype(np.uint8)
    px[rng.random(n) < 0.02] = np.nan
    py[rng.random(n) < 0.01] = np.inf
    px[rng.random(n) < 0.01] += 1e6  # outside the frame
    gvalid = (rng.random(len(w.polys)) > 0.05).astype(np.uint8)
    return px, py, valid, w.polys, gvalid


@pytest.mark.parametrize("kind", ["star", "zipf", "degenerate"])
@pytest.mark.parametrize("n", SIZES)
def test_direct_equals_grouped(vsabi, ctx, kind, n):
    import torch

    px, py, valid, polys, gvalid = _inputs(kind, n)
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda()
           for a in (px, py, valid, polys.x, polys.y, polys.ring_off, polys.part_off, polys.geom_off, gvalid)]
    index = vsabi.DeviceIndex(ctx, vsabi.make_polygons(*dev[3:]), learned=True)
    for pts in (vsabi.make_points(*dev[:3]), vsabi.make_points(*dev[:2])):
        for pred in (vsabi.PRED_WITHIN, vsabi.PRED_INTERSECTS, vsabi.PRED_TOUCHES, vsabi.PRED_BBOX):
            grouped = index.join(pts, pred, vsabi.METHOD_LEARNED, flags=vsabi.JOIN_LEARNED_NO_STAGE)
            direct = index.join(pts, pred, vsabi.METHOD_LEARNED)
            assert torch.equal(direct[0], grouped[0]) and torch.equal(direct[1], grouped[1])
            assert direct[2]["candidates"] == grouped[2]["candidates"]
            left, right, _ = index.join(pts, pred, vsabi.METHOD_LEARNED, sort=False)
            assert set(zip(left.tolist(), right.tolist())) == set(zip(grouped[0].tolist(), grouped[1].tolist()))


def test_direct_capacity(vsabi, ctx):
    """Too small a pair buffer: the required size is reported and nothing beyond the buffer is written."""
    import torch

    px, py, _, polys, _ = _inputs("star", 5_000)
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda()
           for a in (px, py, polys.x, polys.y, polys.ring_off, polys.part_off, polys.geom_off)]
    index = vsabi.DeviceIndex(ctx, vsabi.make_polygons(*dev[2:]), learned=True)
    pts = vsabi.make_points(*dev[:2])
    need = index.join(pts, vsabi.PRED_WITHIN, vsabi.METHOD_LEARNED)[0].numel()
    for cap in (0, 1, need - 1):
        buf = torch.full((2, need + 8), -7, dtype=torch.int32, device="cuda")
        with pytest.raises(vsabi.CapacityError) as err:
            index.join_into(pts, vsabi.PRED_WITHIN, vsabi.METHOD_LEARNED, buf[0][:cap], buf[1][:cap], sort=True)
        assert err.value.required == need
        assert bool((buf[:, cap:] == -7).all())
    # and the next call finds its counters clean
    assert index.join(pts, vsabi.PRED_WITHIN, vsabi.METHOD_LEARNED)[0].numel() == need
