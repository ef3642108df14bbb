"""Keys that a large part of a table has: what the table's flags, the probes of its long bucket and the writing of its
matches cost, and their results at the sizes where the stage divides its items differently, against the oracle."""
import ctypes

import numpy as np
import pytest

import oracle_lib
from test_gpu_scan_forms import check, column

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def plain(pkg):
    """A context that does not replay queries."""
    c = pkg.Context(0)
    c.set_graphs(False)
    yield c
    c.close()


def timed(pkg, ctx, oracle, cp, label):
    """The shortest device time of five runs, the result checked."""
    want = oracle.execute(cp.ref())
    plan = cp.struct
    res = [ctx.upload(plan.inputs[i]) for i in range(plan.num_inputs)]
    try:
        best = 1e9
        for _ in range(5):
            with ctx.execute_resident(cp, res) as r:
                best = min(best, r.stats().device_ms)
                got, keep = r.table_struct()
                oracle_lib.assert_same_rows(oracle, ctypes.byref(got), want.view(), label)
        return best
    finally:
        for x in res:
            x.free()


def ints(pkg, values):
    return column(pkg, pkg.INT32, np.asarray(values, np.int32))


def bucket(keys):
    """The bucket of INT32 keys in a table of 2^20 buckets (in a larger one, keys of two of these are apart too)."""
    return (np.asarray(keys, np.uint64) * np.uint64(0x9E3779B97F4A7C15)) >> np.uint64(44)


def one_key_table(pkg, rows=2_000_000):
    """A table of one key, its rows fed by a probe, probed by a larger one that does not have the key."""
    rng = np.random.default_rng(1)
    i32 = pkg.INT32
    p = pkg.Plan()
    top = rng.integers(100, 1 << 28, rows * 3 // 2)
    top = top[bucket(top) != bucket(7)]
    p.new_input(pkg.ColumnarTable(len(top), [ints(pkg, top), ints(pkg, np.arange(len(top)))]))
    p.new_input(pkg.ColumnarTable(rows, [ints(pkg, np.full(rows, 7)), ints(pkg, np.arange(rows)),
                                         ints(pkg, rng.integers(0, 500, rows))]))
    p.new_input(pkg.ColumnarTable(500, [ints(pkg, np.arange(500))]))
    a = p.new_scan_node(0, [(0, i32), (1, i32)])
    b = p.new_scan_node(1, [(0, i32), (1, i32), (2, i32)])
    fed = p.new_join_node(False, b, p.new_scan_node(2, [(0, i32)]), 2, 0, [(0, i32), (1, i32)])
    p.root = p.new_join_node(False, a, fed, 0, 0, [(1, i32), (3, i32)])
    return pkg.CPlan(p)


def test_flags_of_a_table_of_one_key(pkg, plain, oracle):
    # The flags were one warp's work: 62,500 steps of a load, 20 ms of 22.
    assert timed(pkg, plain, oracle, one_key_table(pkg), "one key") < 10.0


def two_tables(pkg, probe, build):
    """probe(key, row) joined with build(key, row): the build's keys repeat."""
    i32 = pkg.INT32
    p = pkg.Plan()
    p.new_input(pkg.ColumnarTable(len(probe), [ints(pkg, probe), ints(pkg, np.arange(len(probe)))]))
    p.new_input(pkg.ColumnarTable(len(build), [ints(pkg, build), ints(pkg, np.arange(len(build)))]))
    a = p.new_scan_node(0, [(0, i32), (1, i32)])
    b = p.new_scan_node(1, [(0, i32), (1, i32)])
    p.root = p.new_join_node(False, a, b, 0, 0, [(1, i32), (3, i32)])
    return pkg.CPlan(p)


def other_key(pkg):
    # (A build above 131,072 rows has no filter that would drop the probes.)
    keys = np.arange(1, 1 << 24)
    first, other = keys[bucket(keys) == bucket(12345)][:2]  # one bucket
    rng = np.random.default_rng(2)
    build = np.concatenate([np.full(40_000, first), rng.integers(1 << 27, 1 << 28, 100_000)])
    probe = np.full(4_000_000, other)
    probe[:: 500_000] = build[-8:]
    return two_tables(pkg, probe, rng.permutation(build))


def hot_keys(pkg):
    # 2,000 rows that find 1,000 rows each.
    rng = np.random.default_rng(3)
    return two_tables(pkg, np.concatenate([rng.integers(0, 2, 2000), np.arange(10, 1500)]),
                      rng.permutation(np.repeat([0, 1], 1000)))


def test_probes_of_another_keys_bucket(pkg, plain, oracle):
    # Each probe walked the bucket's 40,000 entries by itself: 210 ms.
    assert timed(pkg, plain, oracle, other_key(pkg), "other key") < 70.0


def test_few_rows_with_many_matches(pkg, plain, oracle):
    # All matches were a few blocks' to write, each walking its buckets twice: 1.15 ms.
    assert timed(pkg, plain, oracle, hot_keys(pkg), "hot keys") < 0.5


# Probe rows around a block's and a warp's shares, by the matches of each (a block takes 512 rows, fewer from four matches on):
# `rows` of a table's 10,000 rows pass a first probe and reach the one whose keys repeat.
@pytest.mark.parametrize("copies", [3, 5, 40, 300])
@pytest.mark.parametrize("rows", [1, 7, 8, 9, 63, 65, 255, 257, 511, 513, 1100])
@pytest.mark.parametrize("wide", [False, True])
def test_shares_of_a_block(pkg, ctx, oracle, rows, copies, wide):
    rng = np.random.default_rng(rows * 1000 + copies)
    i32, (kt, kn) = pkg.INT32, (pkg.INT64, np.int64) if wide else (pkg.INT32, np.int32)
    high = (3 << 32) if wide else 0
    passes = rng.permutation(np.concatenate([np.arange(rows), np.arange(20_000, 30_000 - rows)]))
    key = (rng.integers(0, 9, 10_000) | high).astype(kn)  # 0 to 5 are there, each `copies` times
    own = rng.permutation(np.concatenate([np.repeat(np.arange(6), copies), np.arange(100, 300)]) | high).astype(kn)
    p = pkg.Plan()
    p.new_input(pkg.ColumnarTable(10_000, [ints(pkg, passes), column(pkg, kt, key), ints(pkg, np.arange(10_000))]))
    p.new_input(pkg.ColumnarTable(rows, [ints(pkg, rng.permutation(rows))]))
    p.new_input(pkg.ColumnarTable(len(own), [column(pkg, kt, own), ints(pkg, np.arange(len(own)))]))
    a = p.new_scan_node(0, [(0, i32), (1, kt), (2, i32)])
    first = p.new_join_node(False, a, p.new_scan_node(1, [(0, i32)]), 0, 0, [(1, kt), (2, i32)])
    p.root = p.new_join_node(False, first, p.new_scan_node(2, [(0, kt), (1, i32)]), 0, 0, [(1, i32), (3, i32)])
    check(pkg, ctx, oracle, pkg.CPlan(p), f"rows {rows} copies {copies} wide {wide}")


def test_flags_of_many_repeated_keys(pkg, plain, oracle):
    """35,000 keys six times each: every bucket has a repeat to report."""
    rng = np.random.default_rng(4)
    spread = lambda k: k.astype(np.int64) | ((k.astype(np.int64) % 5) << 33)  # noqa: E731
    own = np.repeat(rng.permutation(70_000)[:35_000], 6)
    probe = rng.integers(0, 10_000_000, 400_000)  # (few of them there)
    p = pkg.Plan()
    p.new_input(pkg.ColumnarTable(len(probe), [column(pkg, pkg.INT64, spread(probe)), ints(pkg, np.arange(len(probe)))]))
    p.new_input(pkg.ColumnarTable(len(own), [column(pkg, pkg.INT64, spread(own)), ints(pkg, np.arange(len(own)))]))
    a = p.new_scan_node(0, [(0, pkg.INT64), (1, pkg.INT32)])
    b = p.new_scan_node(1, [(0, pkg.INT64), (1, pkg.INT32)])
    p.root = p.new_join_node(False, a, b, 0, 0, [(1, pkg.INT32), (3, pkg.INT32)])
    best = timed(pkg, plain, oracle, pkg.CPlan(p), "repeated keys")
    # Each bucket stored the one word of the flag: 140 us for that alone, 8 now.
    assert best < 0.15, best
