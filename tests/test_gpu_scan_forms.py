"""The scan-side probe in its forms, against the oracle, at the sizes where
they can go wrong: part groups of 32 rows, part pages, pages with NULLs (their
rows taken by the null bitmap), unit boundaries, tables probed with and
without a filter, the fused unique-key stages, INT32 and INT64 keys."""
import ctypes

import numpy as np
import pytest

import oracle_lib

pytestmark = pytest.mark.gpu


def column(pkg, dtype, values, valid=None):
    values = np.ascontiguousarray(values)
    h = ctypes.c_void_p()
    st = pkg.wlib().bjw_encode_column(dtype, len(values), values.ctypes.data,
                                      None if valid is None else valid.ctypes.data, None, None, ctypes.byref(h))
    assert st == 0
    n, ptrs = pkg.wlib().bjw_pages_count(h), pkg.wlib().bjw_pages_ptrs(h)
    data = b"".join(ctypes.string_at(ptrs[i], 8192) for i in range(n))
    pkg.wlib().bjw_pages_free(h)
    return pkg.Column(dtype, data)


def star(pkg, seed, fact, dims, keep, nulls, wide, copies=1):
    """fact(id, k0, ...) joined with dims[j] keys of which a share `keep` is present, each `copies` times."""
    rng = np.random.default_rng(seed)
    kt, kn = (pkg.INT64, np.int64) if wide else (pkg.INT32, np.int32)
    spread = (lambda k: k.astype(np.int64) | ((k.astype(np.int64) % 8 - 4) << 32)) if wide else \
             (lambda k: (k.astype(np.int64) - 7).astype(np.int32))  # INT32 keys around zero
    p = pkg.Plan()
    cols = [column(pkg, pkg.INT32, np.arange(fact, dtype=np.int32))]
    for d in dims:
        valid = None if not nulls else (rng.random(fact) >= nulls).astype(np.uint8)
        cols.append(column(pkg, kt, spread(rng.integers(0, d, fact)).astype(kn), valid))
    p.new_input(pkg.ColumnarTable(fact, cols))
    left = p.new_scan_node(0, [(0, pkg.INT32)] + [(1 + j, kt) for j in range(len(dims))])
    width = 1 + len(dims)
    for j, d in enumerate(dims):
        own = np.repeat(rng.permutation(d)[:max(1, int(d * keep))], copies)
        t = p.new_input(pkg.ColumnarTable(len(own), [
            column(pkg, kt, spread(own).astype(kn)),
            column(pkg, pkg.INT32, rng.integers(0, 1 << 30, len(own), dtype=np.int32))]))
        right = p.new_scan_node(t, [(0, kt), (1, pkg.INT32)])
        attrs = [(i, pkg.INT32 if i == 0 else kt) for i in range(1 + len(dims))]
        attrs += [(i, pkg.INT32) for i in range(1 + len(dims), width)] + [(width + 1, pkg.INT32)]
        left = p.new_join_node(False, left, right, 1 + j, 0, attrs)
        width += 1
    p.root = left
    return pkg.CPlan(p)


def check(pkg, ctx, oracle, cp, label):
    want = oracle.execute(cp.ref())
    with ctx.execute_raw(cp) as r:
        got, keep = r.table_struct()
        oracle_lib.assert_same_rows(oracle, ctypes.byref(got), want.view(), label + " host")
    plan = cp.struct
    res = [ctx.upload(plan.inputs[i]) for i in range(plan.num_inputs)]
    try:
        for run in range(3):  # recorded, captured, replayed
            with ctx.execute_resident(cp, res) as r:
                got, keep = r.table_struct()
                oracle_lib.assert_same_rows(oracle, ctypes.byref(got), want.view(), f"{label} resident {run}")
    finally:
        for x in res:
            x.free()


# Rows: a lone row, group and batch edges, page edges (1,984 INT32 rows, 1,007 INT64 rows), several pages.
@pytest.mark.parametrize("fact", [1, 31, 33, 127, 128, 129, 1023, 1025, 1007, 1008, 1984, 1985, 4001, 40_003])
@pytest.mark.parametrize("nulls", [0.0, 0.1, 0.9])
@pytest.mark.parametrize("wide", [False, True])
def test_direct_scan(pkg, ctx, oracle, fact, nulls, wide):
    check(pkg, ctx, oracle, star(pkg, fact, fact, [300], 0.5, nulls, wide), f"fact {fact} nulls {nulls} wide {wide}")


@pytest.mark.parametrize("dims", [[500, 200], [4000, 900, 60], [70_000, 5, 300, 20]])
@pytest.mark.parametrize("keep", [0.05, 0.6, 1.0])
@pytest.mark.parametrize("wide", [False, True])
def test_fused_stages(pkg, ctx, oracle, dims, keep, wide):
    check(pkg, ctx, oracle, star(pkg, len(dims), 30_011, dims, keep, 0.05, wide), f"dims {dims} keep {keep}")


# Either side of the line where a filtered scan takes the staged form (512 pages).
@pytest.mark.parametrize("fact", [512 * 1984, 512 * 1984 + 1])
def test_filter_form_line(pkg, ctx, oracle, fact):
    check(pkg, ctx, oracle, star(pkg, 5, fact, [3000, 700], 0.1, 0.0, False), f"fact {fact}")


# Build sizes: bucket counts' edges, the cluster build's last size, the filter's last size, a large build; each key
# once, twice (both keys in the bucket) and seven times (buckets walked); NULL keys and NULL payloads.
@pytest.mark.parametrize("rows", [1, 15, 16, 1025, 4096, 4097, 131_072, 131_073])
@pytest.mark.parametrize("copies", [1, 2, 7])
@pytest.mark.parametrize("wide", [False, True])
def test_builds(pkg, ctx, oracle, rows, copies, wide):
    rng = np.random.default_rng(rows * 10 + copies)
    kt = pkg.INT64 if wide else pkg.INT32
    spread = (lambda k: k.astype(np.int64) | ((k.astype(np.int64) % 8 - 4) << 32)) if wide else \
             (lambda k: (k.astype(np.int64) - 7).astype(np.int32))
    own = rng.permutation(np.repeat(np.arange(-(-rows // copies)), copies)[:rows])
    fact = 150_000 if rows > 5000 else 9_001
    fk = rng.integers(0, 2 * len(own) // copies + 2, fact)
    some = lambda n, p: (rng.random(n) >= p).astype(np.uint8)  # noqa: E731
    p = pkg.Plan()
    p.new_input(pkg.ColumnarTable(fact, [column(pkg, kt, spread(fk)), column(pkg, pkg.INT32, np.arange(fact, dtype=np.int32))]))
    p.new_input(pkg.ColumnarTable(rows, [
        column(pkg, kt, spread(own), some(rows, 0.1)),
        column(pkg, pkg.INT64, rng.integers(0, 1 << 50, rows), some(rows, 0.3)),
        column(pkg, pkg.FP64, rng.random(rows))]))
    a = p.new_scan_node(0, [(0, kt), (1, pkg.INT32)])
    b = p.new_scan_node(1, [(0, kt), (1, pkg.INT64), (2, pkg.FP64)])
    p.root = p.new_join_node(False, a, b, 0, 0, [(0, kt), (1, pkg.INT32), (3, pkg.INT64), (4, pkg.FP64)])
    check(pkg, ctx, oracle, pkg.CPlan(p), f"rows {rows} copies {copies} wide {wide}")


def _lookup(pkg, fact, null_payload):
    """Every fact row finds one row; INT32, INT64 and FP64 results from the fact and from the build."""
    rng = np.random.default_rng(fact)
    valid = (rng.random(97) >= 0.5).astype(np.uint8) if null_payload else None
    p = pkg.Plan()
    p.new_input(pkg.ColumnarTable(fact, [
        column(pkg, pkg.INT32, rng.integers(0, 97, fact, dtype=np.int32)),
        column(pkg, pkg.INT32, np.arange(fact, dtype=np.int32)), column(pkg, pkg.FP64, rng.random(fact))]))
    p.new_input(pkg.ColumnarTable(97, [
        column(pkg, pkg.INT32, rng.permutation(97).astype(np.int32)),
        column(pkg, pkg.INT64, rng.integers(0, 1 << 60, 97), valid),
        column(pkg, pkg.INT32, rng.integers(0, 1 << 30, 97, dtype=np.int32))]))
    a = p.new_scan_node(0, [(0, pkg.INT32), (1, pkg.INT32), (2, pkg.FP64)])
    b = p.new_scan_node(1, [(0, pkg.INT32), (1, pkg.INT64), (2, pkg.INT32)])
    p.root = p.new_join_node(False, a, b, 0, 0, [(0, pkg.INT32), (1, pkg.INT32), (2, pkg.FP64), (4, pkg.INT64),
                                                 (5, pkg.INT32)])
    return pkg.CPlan(p)


# Result sizes: part threads of a page, page edges (1,984 INT32 rows, 1,007 INT64 and FP64 rows), several pages.
@pytest.mark.parametrize("rows", [1, 8, 255, 257, 1007, 1008, 1984, 1985, 2014, 2015, 9000])
@pytest.mark.parametrize("null_payload", [False, True])
def test_result_pages(pkg, ctx, oracle, rows, null_payload):
    check(pkg, ctx, oracle, _lookup(pkg, rows, null_payload), f"rows {rows} null {null_payload}")


@pytest.mark.parametrize("null_payload", [False, True])
def test_device_results_of_replays_in_flight(pkg, oracle, null_payload):
    """Replays write their pages into memory of their own: several in flight, each complete."""
    cp = _lookup(pkg, 5000, null_payload)
    want = oracle.execute(cp.ref())
    with pkg.Context(0) as c:
        res = [c.upload(cp.struct.inputs[i]) for i in range(2)]
        for run in range(2):  # recorded, captured
            c.execute_resident(cp, res, pkg.RESULT_DEVICE).free()
        flying = [c.execute_resident(cp, res, pkg.RESULT_DEVICE | pkg.RESULT_ASYNC) for _ in range(4)]
        at = [pkg.lib().bj_result_device_page(r.handle, 0, 0) for r in flying]
        assert len(set(at)) == 4
        for r in flying:
            r.wait()
            t = pkg.Plan()
            t.new_input(r.to_table())
            got = pkg.CPlan(t)
            oracle_lib.assert_same_rows(oracle, ctypes.byref(got.struct.inputs[0]), want.view(), "device result")
            r.free()
        for x in res:
            x.free()


# Keys that repeat: few, more than a bucket entry's bit mask (33 and more), more matches than a block collects (4,096),
# a stage over a scan's rows and one over items; NULL keys.
@pytest.mark.parametrize("copies,rows", [(2, 3000), (33, 3000), (70, 2100), (400, 800)])
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("dims", [1, 2])
def test_repeated_keys(pkg, ctx, oracle, copies, rows, wide, dims):
    fact = 1300 if dims == 2 and copies > 33 else 5000
    sizes = [rows // copies, 40][:dims]
    check(pkg, ctx, oracle, star(pkg, copies, fact, sizes, 1.0, 0.1, wide, copies if dims == 1 else min(copies, 40)),
          f"copies {copies} wide {wide} dims {dims}")


@pytest.mark.parametrize("fact", [511, 512, 513, 512 * 1984, 512 * 1984 + 1])
def test_repeated_keys_sizes(pkg, ctx, oracle, fact):
    check(pkg, ctx, oracle, star(pkg, fact, fact, [4000], 0.03, 0.0, False, 3), f"fact {fact}")


# Builds fed by probes: sized by the input's rows up to 65,536, by their counted items beyond; none, some and all rows
# surviving; the sub-dimension's keys unique and repeated.
@pytest.mark.parametrize("rows", [1, 300, 65_536, 65_537])
@pytest.mark.parametrize("keep", [0.0, 0.4, 1.0])
@pytest.mark.parametrize("copies", [1, 2])
def test_fed_builds(pkg, ctx, oracle, rows, keep, copies):
    rng = np.random.default_rng(rows + copies)
    fact, sub = (100_003 if rows > 300 else 2003), max(1, rows // 7)
    p = pkg.Plan()
    i32 = lambda v: column(pkg, pkg.INT32, np.asarray(v, dtype=np.int32))  # noqa: E731
    some = (rng.random(rows) >= 0.05).astype(np.uint8)
    p.new_input(pkg.ColumnarTable(fact, [i32(np.arange(fact)), i32(rng.integers(0, rows, fact))]))
    p.new_input(pkg.ColumnarTable(rows, [i32(rng.permutation(rows)),
                                         column(pkg, pkg.INT32, rng.integers(0, sub, rows).astype(np.int32), some)]))
    own = np.repeat(rng.permutation(sub)[:max(1, int(sub * keep))] + (0 if keep else 2 * sub), copies)
    p.new_input(pkg.ColumnarTable(len(own), [i32(own), i32(rng.integers(0, 1 << 30, len(own)))]))
    f = p.new_scan_node(0, [(0, pkg.INT32), (1, pkg.INT32)])
    d = p.new_scan_node(1, [(0, pkg.INT32), (1, pkg.INT32)])
    s = p.new_scan_node(2, [(0, pkg.INT32), (1, pkg.INT32)])
    j = p.new_join_node(False, f, d, 1, 0, [(0, pkg.INT32), (3, pkg.INT32)])
    p.root = p.new_join_node(False, j, s, 1, 0, [(0, pkg.INT32), (3, pkg.INT32)])
    check(pkg, ctx, oracle, pkg.CPlan(p), f"rows {rows} keep {keep} copies {copies}")


# The staged filter over pages with NULLs: survivors find their rows from their values' places (pages of few and of
# many NULLs, all-NULL chunks, a page's last value), over more than 512 pages.
@pytest.mark.parametrize("nulls", [0.02, 0.5, 0.97])
@pytest.mark.parametrize("keep", [0.02, 0.3])
def test_filter_over_nulls(pkg, ctx, oracle, nulls, keep):
    fact = int(1_100_000 / (1 - nulls)) if nulls < 0.9 else 8_000_000
    check(pkg, ctx, oracle, star(pkg, 3, fact, [20_000], keep, nulls, False), f"nulls {nulls} keep {keep}")
