"""Nearest joins where the single walk's tie list (six entries a point, six a
polygon) is full, one short or overflows into the two-walk path; and points as
far away as the FP32 bounds reach."""
import numpy as np
import pytest

from test_gpu_distance import _device, _oracle_polys, syn

pytestmark = pytest.mark.gpu


def _copies(k, seed):
    """300 stars, each present k times: every nearest distance has at least k polygons."""
    w = syn.star_join(seed=seed, n_points=3_000, n_polys=300)
    p = w.polys
    xs, ys, sizes = [], [], []
    for _ in range(k):
        for a, b in zip(p.ring_off[:-1], p.ring_off[1:]):
            xs.append(p.x[a:b])
            ys.append(p.y[a:b])
            sizes.append(b - a)
    polys = syn._rings_to_soa(np.array(sizes), np.concatenate(xs), np.concatenate(ys))
    px = np.concatenate([w.px, [1e12, -1e30, 1e30, np.nan, np.inf]])
    py = np.concatenate([w.py, [-3.0, 1e30, 0.5, 0.5, -np.inf]])
    return syn.Workload(name="copies", px=px, py=py, polys=polys)


@pytest.mark.parametrize("k", [1, 5, 6, 7, 13])
def test_ties_around_the_list_size(ctx, vsabi, oracle, k):
    w = _copies(k, seed=k)
    index, pts, keep = _device(vsabi, ctx, w)
    P = _oracle_polys(oracle, w)
    for md in (np.inf, 0.0, 0.01):
        el, er, ed = oracle.nearest_join(w.px, w.py, None, P, md)
        gl, gr, gd, _ = index.nearest(pts, max_distance=md)
        np.testing.assert_array_equal(gl.cpu().numpy(), el)
        np.testing.assert_array_equal(gr.cpu().numpy(), er)
        np.testing.assert_array_equal(gd.cpu().numpy().view(np.int64), ed.view(np.int64))


@pytest.mark.parametrize("k", [1, 5, 6, 7, 13])
def test_equal_points_around_the_list_size(ctx, vsabi, oracle, k):
    import torch

    w = _copies(1, seed=20 + k)
    px, py = np.tile(w.px[:-5], k), np.tile(w.py[:-5], k)
    dx, dy = torch.from_numpy(px).cuda(), torch.from_numpy(py).cuda()
    pidx = vsabi.point_index(ctx, dx, dy)
    p = w.polys
    t = [torch.from_numpy(np.ascontiguousarray(getattr(p, a))).cuda()
         for a in ("x", "y", "ring_off", "part_off", "geom_off")]
    P = vsabi.make_polygons(*t)
    for md in (np.inf, 0.0, 0.01):
        el, er, ed = oracle.nearest_polygons_join(px, py, None, _oracle_polys(oracle, w), md)
        gl, gr, gd, _ = vsabi.nearest_polygons(ctx, pidx, P, max_distance=md)
        np.testing.assert_array_equal(gl.cpu().numpy(), el)
        np.testing.assert_array_equal(gr.cpu().numpy(), er)
        np.testing.assert_array_equal(gd.cpu().numpy().view(np.int64), ed.view(np.int64))


def _time(f):
    import time

    import torch

    f()
    best = 1e9
    for _ in range(5):
        torch.cuda.synchronize()
        t = time.perf_counter()
        f()
        torch.cuda.synchronize()
        best = min(best, time.perf_counter() - t)
    return best


@pytest.mark.parametrize("k", [5, 6, 7, 12])
@pytest.mark.parametrize("side", ["points", "polygons"])
def test_time_grows_with_the_copies(ctx, vsabi, side, k):
    """Every polygon (point) k times: k times the pairs, for at most five times as much time a pair as without copies,
    also where the single walk leaves some or all queries to the exact walks (a mixture of far-apart queries in their
    packets took 39 times as long for 6 copies of the polygons, 310 for 5 of the points)."""
    import torch

    w = syn.utm_join(seed=3, n_points=150_000, n_polys=5_000)
    q = w.polys

    def run(copies):
        sizes = np.diff(q.ring_off)
        if side == "polygons":
            sizes = np.tile(sizes, copies)
            xs, ys, px, py = np.tile(q.x, copies), np.tile(q.y, copies), w.px, w.py
        else:
            xs, ys, px, py = q.x, q.y, np.tile(w.px[:50_000], copies), np.tile(w.py[:50_000], copies)
        polys = syn._rings_to_soa(sizes, xs, ys)
        t = [torch.from_numpy(np.ascontiguousarray(getattr(polys, a))).cuda()
             for a in ("x", "y", "ring_off", "part_off", "geom_off")]
        P = vsabi.make_polygons(*t)
        dx, dy = torch.from_numpy(px).cuda(), torch.from_numpy(py).cuda()
        if side == "polygons":
            index, pts = vsabi.DeviceIndex(ctx, P), vsabi.make_points(dx, dy)
            return index.nearest(pts)[0].numel(), _time(lambda: index.nearest(pts, sort=False))
        index = vsabi.point_index(ctx, dx, dy)
        return (vsabi.nearest_polygons(ctx, index, P)[0].numel(),
                _time(lambda: vsabi.nearest_polygons(ctx, index, P, sort=False)))

    pairs_one, one = run(1)
    pairs, many = run(k)
    assert pairs == k * pairs_one
    print(side, k, one, many, many / one)
    assert many < 5 * k * one, (one, many)


def _crowd(seed):
    """3000 stars, about 20 over any place and some of them twice; points anywhere, on vertices, beside edges (an ulp
    off, where a distance may round to 0) and outside them all."""
    rng = np.random.default_rng(seed)
    p = syn.star_polygons(rng, 3_000, 0.0, 250.0)
    k = rng.choice(3_000, 400, replace=False)
    xs, ys, sizes = [p.x], [p.y], [np.diff(p.ring_off)]
    for g in k:
        xs.append(p.x[p.ring_off[g]:p.ring_off[g + 1]])
        ys.append(p.y[p.ring_off[g]:p.ring_off[g + 1]])
        sizes.append([p.ring_off[g + 1] - p.ring_off[g]])
    polys = syn._rings_to_soa(np.concatenate(sizes), np.concatenate(xs), np.concatenate(ys))
    v = rng.integers(0, len(p.x) - 1, 600)
    mid_x, mid_y = 0.5 * (p.x[v] + p.x[v + 1]), 0.5 * (p.y[v] + p.y[v + 1])
    px = np.concatenate([rng.uniform(-40, 290, 1500), p.x[v], np.nextafter(p.x[v], 1e9), mid_x, np.nextafter(mid_x, 0)])
    py = np.concatenate([rng.uniform(-40, 290, 1500), p.y[v], p.y[v], mid_y, mid_y])
    return syn.Workload(name="crowd", px=px, py=py, polys=polys)


@pytest.mark.parametrize("max_distance", [np.inf, 0.0, 0.5])
def test_points_under_many_polygons(ctx, vsabi, oracle, max_distance):
    w = _crowd(11)
    index, pts, keep = _device(vsabi, ctx, w)
    el, er, ed = oracle.nearest_join(w.px, w.py, None, _oracle_polys(oracle, w), max_distance)
    gl, gr, gd, _ = index.nearest(pts, max_distance=max_distance)
    np.testing.assert_array_equal(gl.cpu().numpy(), el)
    np.testing.assert_array_equal(gr.cpu().numpy(), er)
    np.testing.assert_array_equal(gd.cpu().numpy().view(np.int64), ed.view(np.int64))


@pytest.mark.parametrize("max_distance", [np.inf, 0.0, 0.5])
def test_polygons_over_many_points(ctx, vsabi, oracle, max_distance):
    import torch

    w = _crowd(12)
    px, py = np.concatenate([w.px, w.px[::3]]), np.concatenate([w.py, w.py[::3]])
    dx, dy = torch.from_numpy(px).cuda(), torch.from_numpy(py).cuda()
    pidx = vsabi.point_index(ctx, dx, dy)
    t = [torch.from_numpy(np.ascontiguousarray(getattr(w.polys, a))).cuda()
         for a in ("x", "y", "ring_off", "part_off", "geom_off")]
    el, er, ed = oracle.nearest_polygons_join(px, py, None, _oracle_polys(oracle, w), max_distance)
    gl, gr, gd, _ = vsabi.nearest_polygons(ctx, pidx, vsabi.make_polygons(*t), max_distance=max_distance)
    np.testing.assert_array_equal(gl.cpu().numpy(), el)
    np.testing.assert_array_equal(gr.cpu().numpy(), er)
    np.testing.assert_array_equal(gd.cpu().numpy().view(np.int64), ed.view(np.int64))
