"""What the bounded waits inside kernels leave behind when they run out.

Such a wait ends in practice long before its limit, so these tests build the library once more with the limit of a
source file lowered, and use that library in a process of its own."""
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

import pytest

from vibespatial_b200 import _build

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent


def _library(folder, defines):
    """The library with -D options for some sources (name -> options); the other sources' objects are the build's,
    where it left them."""
    cxx = ["-ccbin", "/usr/bin/g++"] if Path("/usr/bin/g++").exists() else []
    base = [_build.nvcc(), *_build.NVCC_FLAGS, *cxx]

    def compile_one(src):
        kept = ROOT / "_build" / (src.stem + ".o")
        newest = max(p.stat().st_mtime for p in (src, *src.parent.glob("*.cuh"), ROOT / "include" / "vsjoin.h"))
        if src.stem not in defines and kept.exists() and kept.stat().st_mtime >= newest:
            return str(kept)
        obj = folder / (src.stem + ".o")
        subprocess.run([*base, *defines.get(src.stem, ()), "-c", str(src), "-o", str(obj), "-I",
                        str(_build.INCLUDE)], check=True, capture_output=True, text=True)
        return str(obj)

    with ThreadPoolExecutor(4) as pool:
        objs = list(pool.map(compile_one, _build.sources()))
    lib = folder / "libvsjoin_waits.so"
    subprocess.run([*base, "-shared", "-o", str(lib), *objs, "-lcudart"], check=True, capture_output=True, text=True)
    return lib


def _run(lib, code):
    head = (f"import sys\nsys.path.insert(0, {str(ROOT)!r})\nimport numpy as np\nimport torch\n"
            f"from vibespatial_b200 import _abi\n_abi._lib = _abi.load({str(lib)!r})\n"
            "from vibespatial_b200.testing import synthetic as syn\nctx = _abi.default_context(0)\n"
            "dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()\n")
    r = subprocess.run([sys.executable, "-c", head + code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    print(r.stdout)


needs_nvcc = pytest.mark.skipif(shutil.which(_build.nvcc()) is None, reason="needs nvcc")


@needs_nvcc
def test_sorts_whose_tiles_do_not_wait(tmp_path):
    """A pass whose tiles give their earlier ones one poll each counts those tiles' keys itself: same order, whatever
    the tile and digit sizes (keys with values; pairs by runs and by all digits), and no status to lose."""
    lib = _library(tmp_path, {"primitives": ["-DVS_SORT_WAIT_LIMIT=1"]})
    _run(lib, """
for n in (8193, 9217, 303_104, 303_105, 400_003):
    rng = np.random.default_rng(n)
    for bits in (24, 64):
        keys = rng.integers(0, 2**63, n, dtype=np.uint64) & np.uint64(2**bits - 1)
        keys[n // 2:] = keys[: n - n // 2]
        dk, dv = dev(keys.view(np.int64)), dev(np.arange(n, dtype=np.int32))
        _abi.radix_sort_pairs(ctx, dk, dv, bits)
        order = np.argsort(keys, kind="stable")
        assert np.array_equal(dk.cpu().numpy().view(np.uint64), keys[order]), (n, bits)
        assert np.array_equal(dv.cpu().numpy(), order.astype(np.int32)), (n, bits)
    for rows in (n // 3, 5):
        left, right = (rng.integers(0, h, n).astype(np.int32) for h in (rows, 100_000))
        dl, dr = dev(left), dev(right)
        _abi.sort_pairs(ctx, dl, dr)
        order = np.lexsort((right, left))
        assert np.array_equal(dl.cpu().numpy(), left[order]) and np.array_equal(dr.cpu().numpy(), right[order]), n
w = syn.star_join(seed=3, n_points=100_007, n_polys=2_000)  # rows below 2^17: 9-bit digits
polys = [dev(getattr(w.polys, k)) for k in ("x", "y", "ring_off", "part_off", "geom_off")]
dx, dy = dev(w.px), dev(w.py)
index = _abi.DeviceIndex(ctx, _abi.make_polygons(*polys), learned=True)
tree, cells = (index.join(_abi.make_points(dx, dy), _abi.PRED_WITHIN, m, sort=True)
               for m in (_abi.METHOD_RTREE, _abi.METHOD_LEARNED))
order = np.lexsort((tree[1].cpu().numpy(), tree[0].cpu().numpy()))
assert np.array_equal(order, np.arange(len(order)))
assert torch.equal(tree[0], cells[0]) and torch.equal(tree[1], cells[1])
""")


@needs_nvcc
def test_training_that_gives_up_reports_it(tmp_path):
    """A training whose grid barrier runs out leaves a model that the passes after it can use within their arrays; the
    build then reports the timeout, and the context serves the next calls."""
    lib = _library(tmp_path, {"learned": ["-DVS_TRAIN_WAIT_LIMIT=1"]})
    _run(lib, """
w = syn.star_join(seed=3, n_points=20_003, n_polys=20_000)  # over 16384 cells: 128 blocks
polys = [dev(getattr(w.polys, k)) for k in ("x", "y", "ring_off", "part_off", "geom_off")]
for _ in range(2):
    try:
        _abi.DeviceIndex(ctx, _abi.make_polygons(*polys), learned=True)
        raise SystemExit("no timeout")
    except _abi.VsError as e:
        assert e.status == _abi.VS_E_TIMEOUT and "RMI training" in str(e), e
tree = _abi.DeviceIndex(ctx, _abi.make_polygons(*polys))
dx, dy = dev(w.px), dev(w.py)
pts = _abi.make_points(dx, dy)
left, right, _ = tree.join(pts, _abi.PRED_WITHIN, _abi.METHOD_RTREE)
brute = tree.join(pts, _abi.PRED_WITHIN, _abi.METHOD_BRUTE)
assert left.numel() > 0 and torch.equal(left, brute[0]) and torch.equal(right, brute[1])
""")


@needs_nvcc
@pytest.mark.parametrize("blocks", [1, 7])
def test_training_in_fewer_blocks(tmp_path, blocks):
    """Training blocks that take turns at the samples (a GPU that holds fewer of them) end in a model as good (its
    gradients differ in the order of their FP32 sums only: the lookup windows within 1% of each other) and in the
    pairs of the tree."""
    lib = _library(tmp_path, {"learned": [f"-DVS_TRAIN_BLOCKS={blocks}"]})
    _run(lib, f"""
few, whole = _abi._lib, _abi.load({str(_build.LIB)!r})
w = syn.utm_join(seed=3, n_points=400_003, n_polys=30_000)  # over 16384 cells: 128 lots of samples
polys = [dev(getattr(w.polys, k)) for k in ("x", "y", "ring_off", "part_off", "geom_off")]
dx, dy = dev(w.px), dev(w.py)
pts = _abi.make_points(dx, dy)
index = _abi.DeviceIndex(ctx, _abi.make_polygons(*polys), learned=True)
for flags in (0, _abi.JOIN_LEARNED_NO_STAGE):
    left, right, _ = index.join(pts, _abi.PRED_WITHIN, _abi.METHOD_LEARNED, flags=flags)
    tree = index.join(pts, _abi.PRED_WITHIN, _abi.METHOD_RTREE)
    assert left.numel() > 0 and torch.equal(left, tree[0]) and torch.equal(right, tree[1])
window = index.info()["rmi_mean_window"]
index.close()
_abi._lib = whole
expected = _abi.DeviceIndex(_abi.Context(0), _abi.make_polygons(*polys), learned=True).info()["rmi_mean_window"]
print("windows", window, expected)
assert expected > 4 and abs(window - expected) < 0.01 * expected, (window, expected)
""")
