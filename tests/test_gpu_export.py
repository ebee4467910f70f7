"""Join export on the device (vs_join_export) against the host export
(sjoin._join_indexers on numpy arrays, the reference's _adjust_join_indexers
steps): identical output rows and source pairs for every ``how``, with and
without attribute codes."""
import importlib

import numpy as np
import pytest

vs_sjoin = importlib.import_module("vibespatial_b200.sjoin")

pytestmark = pytest.mark.gpu


def _pairs(rng, n_left, n_right, n_pairs):
    l = rng.integers(0, n_left, n_pairs)
    r = rng.integers(0, n_right, n_pairs)
    u = np.unique(l.astype(np.int64) * n_right + r)
    return (u // n_right).astype(np.int32), (u % n_right).astype(np.int32)


def _codes(rng, n, k, miss=0.1):
    c = rng.integers(0, k, n).astype(np.int64)
    c[rng.random(n) < miss] = -1
    return c


@pytest.mark.parametrize("how", ["inner", "left", "right", "outer"])
@pytest.mark.parametrize("with_codes", [False, True])
# sizes: (left rows, right rows, pairs drawn); the export writes tiles of 2048
# driving rows, so the cases cross tile edges (4096, 2049 rows) and give
# single driving rows thousands of pairs (3 right rows, 20k pairs)
@pytest.mark.parametrize("sizes", [(1000, 300, 5000), (50_000, 20_000, 400_000), (7, 5, 0), (0, 9, 0), (5, 0, 0),
                                   (3000, 3, 20_000), (4096, 2049, 30_000), (2049, 1, 2049)])
def test_export_matches_host(ctx, vsabi, how, with_codes, sizes):
    import torch

    n_left, n_right, n_pairs = sizes
    rng = np.random.default_rng(n_left + 7 * n_right + n_pairs)
    l, r = _pairs(rng, max(n_left, 1), max(n_right, 1), n_pairs) if n_left and n_right else (
        np.zeros(0, np.int32), np.zeros(0, np.int32))
    codes = (_codes(rng, n_left, 5), _codes(rng, n_right, 5)) if with_codes else None
    el, er, es = vs_sjoin._join_indexers(l, r, n_left, n_right, how, codes)
    dl = torch.from_numpy(l).cuda()
    dr = torch.from_numpy(r).cuda()
    lc = None if codes is None else torch.from_numpy(codes[0]).cuda()
    rc = None if codes is None else torch.from_numpy(codes[1]).cuda()
    gl, gr, gs = vsabi.join_export(ctx, dl, dr, n_left, n_right, how, lc, rc)
    np.testing.assert_array_equal(gl.cpu().numpy(), el)
    np.testing.assert_array_equal(gr.cpu().numpy(), er)
    np.testing.assert_array_equal(gs.cpu().numpy(), es)


def test_export_rejects_out_of_range_pairs(ctx, vsabi):
    import torch

    l = torch.tensor([0, 1, 5], dtype=torch.int32, device="cuda")
    r = torch.tensor([0, 0, 0], dtype=torch.int32, device="cuda")
    with pytest.raises(ValueError):
        vsabi.join_export(ctx, l, r, 3, 2, "left")
    with pytest.raises(ValueError):
        vsabi.join_export(ctx, l[:2], r[:2], 3, 2, "left", torch.zeros(3, dtype=torch.int64, device="cuda"))
    # with codes on both sides the attribute filter checks the ranges
    codes_l = torch.zeros(3, dtype=torch.int64, device="cuda")
    codes_r = torch.zeros(2, dtype=torch.int64, device="cuda")
    with pytest.raises(ValueError):
        vsabi.join_export(ctx, l, r, 3, 2, "left", codes_l, codes_r)
    with pytest.raises(ValueError):
        vsabi.join_export(ctx, l[:2], r[:2] - 1, 3, 2, "inner", codes_l, codes_r)


@pytest.mark.parametrize("how", ["left", "right", "outer"])
def test_export_orders_unsorted_pairs(ctx, vsabi, how):
    """Pairs that do not come sorted give the rows of the sorted ones, with their own source positions."""
    import torch

    rng = np.random.default_rng(5)
    l, r = _pairs(rng, 9_000, 700, 20_000)
    el, er, es = vs_sjoin._join_indexers(l, r, 9_000, 700, how, None)
    mix = rng.permutation(len(l))
    gl, gr, gs = (t.cpu().numpy() for t in vsabi.join_export(ctx, torch.from_numpy(l[mix]).cuda(),
                                                             torch.from_numpy(r[mix]).cuda(), 9_000, 700, how))
    np.testing.assert_array_equal(gl, el)
    np.testing.assert_array_equal(gr, er)
    np.testing.assert_array_equal(np.where(gs >= 0, mix[np.maximum(gs, 0)], -1), es)


@pytest.mark.parametrize("n_pairs", [2047, 2048, 2049, 65_536, 200_003])
def test_export_filter_tiles(ctx, vsabi, n_pairs):
    """The one-pass attribute filter at the edges of its tiles of 2048 pairs."""
    import torch

    rng = np.random.default_rng(n_pairs)
    l, r = _pairs(rng, 50_000, 3_000, n_pairs + n_pairs // 8)
    l, r = l[:n_pairs], r[:n_pairs]
    codes = (_codes(rng, 50_000, 3), _codes(rng, 3_000, 3))
    el, er, es = vs_sjoin._join_indexers(l, r, 50_000, 3_000, "inner", codes)
    dev = [torch.from_numpy(a).cuda() for a in (l, r, *codes)]
    gl, gr, gs = vsabi.join_export(ctx, dev[0], dev[1], 50_000, 3_000, "inner", dev[2], dev[3])
    np.testing.assert_array_equal(gl.cpu().numpy(), el)
    np.testing.assert_array_equal(gr.cpu().numpy(), er)
    np.testing.assert_array_equal(gs.cpu().numpy(), es)


def _nonzero_device_memory():
    """Small device allocations full of ones, every other one given back: the context's own words then lie in one of
    these.  Returns what frees the rest."""
    import ctypes

    import torch

    torch.zeros(1, device="cuda")
    rt = ctypes.CDLL("libcudart.so.12")
    blocks = []
    for _ in range(64):
        p = ctypes.c_void_p()
        assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(512)) == 0
        assert rt.cudaMemset(p, 0xFF, ctypes.c_size_t(512)) == 0
        blocks.append(p)
    assert rt.cudaDeviceSynchronize() == 0
    for p in blocks[1::2]:
        assert rt.cudaFree(p) == 0
    return lambda: [rt.cudaFree(p) for p in blocks[::2]]


@pytest.mark.parametrize("n", [0, 5])
def test_export_right_without_kept_pairs_on_a_new_context(vsabi, n):
    """The first call of a context, with no pairs or with all of them filtered out: nothing is sorted, and no status
    is read that nothing has set."""
    import torch

    free = _nonzero_device_memory()
    new = vsabi.Context(0)
    l = torch.arange(n, dtype=torch.int32, device="cuda")
    codes = torch.zeros(8, dtype=torch.int64, device="cuda"), torch.ones(8, dtype=torch.int64, device="cuda")
    gl, gr, gs = vsabi.join_export(new, l, l, 8, 8, "right", *codes)
    assert gl.tolist() == [-1] * 8 and gr.tolist() == list(range(8)) and gs.tolist() == [-1] * 8
    new.close()
    free()


def test_export_of_shuffled_pairs_over_many_tiles(ctx, vsabi):
    """Pairs in any order: the rows of the sorted ones, in time linear in the pairs (20M left rows are 9766 tiles;
    work that grew with pairs x tiles took over 100 times the sorted call, the sort of the pairs takes a few)."""
    import time

    import torch

    n_left, n_right = 20_000_000, 1_000
    rng = np.random.default_rng(8)
    l, r = _pairs(rng, n_left, n_right, 2_000_000)
    mix = rng.permutation(len(l))
    dl, dr = torch.from_numpy(l).cuda(), torch.from_numpy(r).cuda()
    dm = torch.from_numpy(mix).cuda()
    ml, mr = dl[dm], dr[dm]

    def timed(a, b):
        out, best = None, 1e9
        for _ in range(3):
            torch.cuda.synchronize()
            t = time.perf_counter()
            out = vsabi.join_export(ctx, a, b, n_left, n_right, "left")
            torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t)
        return out, best

    (sl, sr, ss), t_sorted = timed(dl, dr)
    (gl, gr, gs), t_mixed = timed(ml, mr)
    assert torch.equal(gl, sl) and torch.equal(gr, sr)
    assert torch.equal(torch.where(gs >= 0, dm[gs.clamp(min=0)], gs), ss)
    assert t_mixed < 20 * t_sorted, (t_mixed, t_sorted)


@pytest.mark.parametrize("how", ["left", "right", "outer"])
@pytest.mark.parametrize("rows", [3, 2048, 2049, 5000])
def test_export_tiles_of_many_pairs(ctx, vsabi, how, rows):
    """Tiles whose pairs several blocks write (from 32768 pairs a tile on), up to more than one of them, with most
    pairs in a few rows and some rows without."""
    import torch

    rng = np.random.default_rng(rows)
    l = np.minimum(rng.integers(0, rows, 700_000), rng.integers(0, rows, 700_000))
    r = rng.integers(0, 90_000, 700_000)
    u = np.unique(l.astype(np.int64) * 90_000 + r)
    u = u[u // 90_000 % 7 != 3]
    l, r = (u // 90_000).astype(np.int32), (u % 90_000).astype(np.int32)
    n_left, n_right = (rows, 90_000) if how != "right" else (90_000, rows)
    if how == "right":
        l, r = r, l
        o = np.lexsort((r, l))
        l, r = l[o], r[o]
    el, er, es = vs_sjoin._join_indexers(l, r, n_left, n_right, how, None)
    gl, gr, gs = vsabi.join_export(ctx, torch.from_numpy(l).cuda(), torch.from_numpy(r).cuda(), n_left, n_right, how)
    np.testing.assert_array_equal(gl.cpu().numpy(), el)
    np.testing.assert_array_equal(gr.cpu().numpy(), er)
    np.testing.assert_array_equal(gs.cpu().numpy(), es)
