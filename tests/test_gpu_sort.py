"""The radix sorts at the sizes where their paths change: one block up to 2048
and 8192 items, tiles of 1024 up to 303104, then tiles of 4096 (pairs) or 3072
(64-bit keys with values); pairs by runs of equal left rows, or by all digits
where rows have many pairs (on average, or one row more than 1024)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 33, 2047, 2048, 2049, 8191, 8192, 8193, 1024 * 9, 1024 * 9 + 1, 303_104, 303_105, 4096 * 80 + 7]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("rows", ["random", "equal", "one_digit", "wide", "short_runs", "long_run", "few_left"])
def test_pairs(vsabi, ctx, n, rows):
    import torch

    rng = np.random.default_rng(n)
    hi = {"random": (50_000_000, 1_000_000), "equal": (1, 1), "one_digit": (1, 200), "wide": (2**31 - 1, 2**31 - 1),
          "short_runs": (max(1, n // 5), 1000), "long_run": (n, 5000), "few_left": (3, 2**20)}
    left, right = (rng.integers(0, h, n).astype(np.int32) for h in hi[rows])
    if rows == "long_run":
        left[: min(n, 3000)] = n // 2
        rng.shuffle(left)
    dl, dr = torch.from_numpy(left).cuda(), torch.from_numpy(right).cuda()
    vsabi.sort_pairs(ctx, dl, dr)
    order = np.lexsort((right, left))
    assert np.array_equal(dl.cpu().numpy(), left[order])
    assert np.array_equal(dr.cpu().numpy(), right[order])


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("bits", [8, 13, 40, 64])
def test_keys_with_values_are_stable(vsabi, ctx, n, bits):
    import torch

    rng = np.random.default_rng(n + bits)
    keys = rng.integers(0, 2**63, n, dtype=np.uint64) & np.uint64(2**bits - 1)
    keys[n // 2:] = keys[: n - n // 2]  # equal keys keep their order
    vals = np.arange(n, dtype=np.int32)
    dk, dv = torch.from_numpy(keys.view(np.int64)).cuda(), torch.from_numpy(vals).cuda()
    vsabi.radix_sort_pairs(ctx, dk, dv, bits)
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(dk.cpu().numpy().view(np.uint64), keys[order])
    assert np.array_equal(dv.cpu().numpy(), vals[order])


def test_join_order(vsabi, ctx, oracle):
    """A sorted join's pairs (left rows below 2^19: 8-bit digits) equal the sorted unsorted join's."""
    import torch

    from vibespatial_b200.testing import synthetic as syn

    w = syn.star_join(seed=3, n_points=300_007, n_polys=2_000)
    dx, dy = torch.from_numpy(w.px).cuda(), torch.from_numpy(w.py).cuda()
    t = {k: torch.from_numpy(getattr(w.polys, k)).cuda() for k in ("x", "y", "ring_off", "part_off", "geom_off")}
    idx = vsabi.DeviceIndex(ctx, vsabi.make_polygons(*t.values()), learned=True)
    pts = vsabi.make_points(dx, dy)
    left, right, _ = idx.join(pts, vsabi.PRED_WITHIN, vsabi.METHOD_LEARNED, sort=True)
    ul, ur, _ = idx.join(pts, vsabi.PRED_WITHIN, vsabi.METHOD_LEARNED, sort=False)
    ul, ur = ul.cpu().numpy(), ur.cpu().numpy()
    order = np.lexsort((ur, ul))
    assert np.array_equal(left.cpu().numpy(), ul[order])
    assert np.array_equal(right.cpu().numpy(), ur[order])


@pytest.mark.parametrize("n", [8_193, 100_003, 400_001])
@pytest.mark.parametrize("run", [3, 31, 32, 33, 63, 64, 65, 100, 129, 700, 1023, 1024, 1025, 3000])
@pytest.mark.parametrize("share", [1.0, 0.5])
def test_runs_of_equal_left_rows(vsabi, ctx, n, run, share):
    """Runs of equal left rows, ordered by their right rows (some equal) where left rows have few pairs on average: as
    long as a warp, two, what a tile holds of its neighbours, and up to the limit and beyond; every pair in one, or
    half of them alone in theirs, so that runs of both kinds share warps and cross tiles."""
    import torch

    rng = np.random.default_rng(n + run)
    in_runs = int(n * share) // run * run
    left = np.concatenate([np.repeat(rng.choice(2**22, in_runs // run, replace=False), run),
                           rng.integers(0, 2**22, n - in_runs)]).astype(np.int32)
    right = rng.integers(0, 500, n).astype(np.int32)
    left[-1] = 2**22  # (few pairs a left row)
    mix = rng.permutation(n)
    left, right = left[mix], right[mix]
    dl, dr = torch.from_numpy(left).cuda(), torch.from_numpy(right).cuda()
    vsabi.sort_pairs(ctx, dl, dr)
    order = np.lexsort((right, left))
    assert np.array_equal(dl.cpu().numpy(), left[order])
    assert np.array_equal(dr.cpu().numpy(), right[order])


def _squares(n_points, counts):
    """A join of n_points points with one square for each count, which holds that many of them (the first ones of a
    fixed order, so that the squares share points)."""
    from vibespatial_b200.testing import synthetic as syn

    rng = np.random.default_rng(n_points)
    at = rng.permutation(n_points)
    px = np.empty(n_points)
    px[at] = np.arange(n_points) + 0.5
    half = np.asarray(counts, np.float64)
    xs = np.stack([0 * half, half, half, 0 * half, 0 * half], 1).ravel()
    ys = np.tile([0.0, 0.0, 1.0, 1.0, 0.0], len(half))
    return px, np.full(n_points, 0.5), syn._rings_to_soa(np.full(len(half), 5), xs, ys)


def _joined(vsabi, ctx, px, py, p):
    import torch

    dx, dy = torch.from_numpy(px).cuda(), torch.from_numpy(py).cuda()
    t = [torch.from_numpy(getattr(p, k)).cuda() for k in ("x", "y", "ring_off", "part_off", "geom_off")]
    idx = vsabi.DeviceIndex(ctx, vsabi.make_polygons(*t))
    pts = vsabi.make_points(dx, dy)
    got = [v.cpu().numpy() for v in idx.join(pts, vsabi.PRED_WITHIN, vsabi.METHOD_RTREE, sort=True)[:2]]
    left, right = (v.cpu().numpy() for v in idx.join(pts, vsabi.PRED_WITHIN, vsabi.METHOD_RTREE, sort=False)[:2])
    order = np.lexsort((right, left))
    assert np.array_equal(got[0], left[order])
    assert np.array_equal(got[1], right[order])
    return len(left)


# left rows of 17, 18, 25 and 26 bits: 9-bit digits; of 24: 8-bit ones
@pytest.mark.parametrize("n_points", [100_007, 262_143, 2**24 + 1, 2**25 + 5, 2**23 + 3])
# the edges of the small sort, of tiles of 1024 and 4096 pairs, and where the latter begin
@pytest.mark.parametrize("pairs", [8_192, 8_193, 9 * 1024, 9 * 1024 + 1, 303_104, 303_105, 4096 * 80 - 1, 4096 * 80 + 1])
def test_join_order_with_a_known_row_count(vsabi, ctx, n_points, pairs):
    """The pairs of a join, whose point count tells the bits of their left rows, sorted by runs of left rows."""
    each = pairs // 4
    assert _joined(vsabi, ctx, *_squares(n_points, [each, each, each, pairs - 3 * each])) == pairs


def test_join_order_with_one_row_of_many_pairs(vsabi, ctx):
    """Few pairs a row on average, but some rows with more than the run pass orders: sorted again by all digits."""
    n = 100_007
    pairs = _joined(vsabi, ctx, *_squares(n, [n] * 2 + [7] * 3_500))
    assert pairs == 2 * n + 7 * 3_500 and pairs < 8 * n
