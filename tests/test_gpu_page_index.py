"""The page index at the sizes where its warps end: columns of one page to
several blocks of pages, and of more pages than a warp takes one by one; bitmap
words at a page's last rows; a bad bitmap, offset or run in a page that is not a
warp's first."""
import numpy as np
import pytest

from test_gpu_scan_forms import check, column

pytestmark = pytest.mark.gpu


def _plan(pkg, key, payload, rows):
    p = pkg.Plan()
    p.new_input(pkg.ColumnarTable(rows, [key, payload]))
    own = np.arange(50, dtype=np.int32)
    p.new_input(pkg.ColumnarTable(50, [column(pkg, pkg.INT32, own), column(pkg, pkg.INT32, own * 3)]))
    a = p.new_scan_node(0, [(0, pkg.INT32), (1, payload.type)])
    b = p.new_scan_node(1, [(0, pkg.INT32), (1, pkg.INT32)])
    p.root = p.new_join_node(False, a, b, 0, 0, [(1, payload.type), (3, pkg.INT32)])
    return p


@pytest.mark.parametrize("rows", [1, 31, 33, 2000, 7 * 2100, 8 * 1984, 8 * 1984 + 1, 60_000])
@pytest.mark.parametrize("nulls", [0.0, 0.2, 1.0])
def test_fixed_width(pkg, ctx, oracle, rows, nulls):
    rng = np.random.default_rng(rows)
    some = lambda: (rng.random(rows) >= nulls).astype(np.uint8)  # noqa: E731
    key = column(pkg, pkg.INT32, rng.integers(0, 80, rows).astype(np.int32), some())
    check(pkg, ctx, oracle, pkg.CPlan(_plan(pkg, key, column(pkg, pkg.FP64, rng.random(rows), some()), rows)),
          f"rows {rows} nulls {nulls}")


def test_many_pages(pkg, ctx, oracle):
    """More pages than a warp each: four a warp (4,737 pages and up)."""
    rows, rng = 4_800 * 1984 + 7, np.random.default_rng(1)
    some = (rng.random(rows) >= 0.001).astype(np.uint8)
    key = column(pkg, pkg.INT32, rng.integers(0, 50_000, rows).astype(np.int32), some)
    check(pkg, ctx, oracle, pkg.CPlan(_plan(pkg, key, column(pkg, pkg.INT32, np.arange(rows, dtype=np.int32)), rows)),
          "many pages")


@pytest.mark.parametrize("rows", [1, 33, 400, 3000])
@pytest.mark.parametrize("nulls", [0.0, 0.3])
def test_strings(pkg, ctx, oracle, rows, nulls):
    rng = np.random.default_rng(rows)
    words = [None if rng.random() < nulls else "x" * int(rng.integers(0, 60)) + str(i) for i in range(rows)]
    if rows > 100:
        words[rows // 2] = "long" * 5000
    key = column(pkg, pkg.INT32, rng.integers(0, 80, rows).astype(np.int32))
    check(pkg, ctx, oracle, pkg.CPlan(_plan(pkg, key, pkg.encode_column(pkg.VARCHAR, words), rows)),
          f"rows {rows} nulls {nulls}")


@pytest.mark.parametrize("page", [0, 3, 9])
@pytest.mark.parametrize("what", ["bitmap", "offsets"])
def test_bad_pages_are_rejected(pkg, ctx, page, what):
    rows, rng = 40_000, np.random.default_rng(2)
    if what == "bitmap":
        some = (rng.random(rows) >= 0.1).astype(np.uint8)
        payload = column(pkg, pkg.INT32, np.arange(rows, dtype=np.int32), some)
        at, value = page * 8192 + 8190, None  # one more (or fewer) row flagged
    else:
        payload = pkg.encode_column(pkg.VARCHAR, ["ab" + str(i) for i in range(rows)])
        at, value = page * 8192 + 4 + 2 * 40, b"\xff\x7f"  # an end offset above the next one
    data = bytearray(payload.data)
    if value:
        data[at:at + 2] = value
    else:
        data[at] ^= 0x10
    key = column(pkg, pkg.INT32, rng.integers(0, 80, rows).astype(np.int32))
    cp = pkg.CPlan(_plan(pkg, key, pkg.Column(payload.type, bytes(data)), rows))
    with pytest.raises(pkg.EngineError) as e:
        ctx.execute_raw(cp)
    assert e.value.status == 1
