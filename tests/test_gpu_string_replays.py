"""Replayed queries with VARCHAR results: their rows come in another order each time, and the pages have to be as many as in
the recording. Rows whose page count by the plain rule depends on which is last, and strings of several pages."""
import ctypes

import numpy as np
import pytest

import oracle_lib
from test_gpu_scan_forms import column

pytestmark = pytest.mark.gpu


def names(pkg, words, seed):
    """fact(key, id) joined with a table of a name a key: every row of the fact comes back."""
    rng = np.random.default_rng(seed)
    n, i32 = len(words), pkg.INT32
    p = pkg.Plan()
    key = rng.permutation(n).astype(np.int32)
    p.new_input(pkg.ColumnarTable(n, [column(pkg, i32, key), column(pkg, i32, np.arange(n, dtype=np.int32)),
                                      pkg.encode_column(pkg.VARCHAR, words)]))
    own = np.arange(n + 50, dtype=np.int32)
    p.new_input(pkg.ColumnarTable(len(own), [column(pkg, i32, rng.permutation(own)), column(pkg, i32, own)]))
    a, b = p.new_scan_node(0, [(0, i32), (1, i32), (2, pkg.VARCHAR)]), p.new_scan_node(1, [(0, i32), (1, i32)])
    p.root = p.new_join_node(False, a, b, 0, 0, [(2, pkg.VARCHAR), (1, i32), (4, i32)])
    return pkg.CPlan(p)


def run(pkg, ctx, oracle, cp, label, times):
    want = oracle.execute(cp.ref())
    res = [ctx.upload(cp.struct.inputs[i]) for i in range(cp.struct.num_inputs)]
    try:
        for k in range(times):
            with ctx.execute_resident(cp, res) as r:
                got, keep = r.table_struct()
                oracle_lib.assert_same_rows(oracle, ctypes.byref(got), want.view(), f"{label} run {k}")
    finally:
        for x in res:
            x.free()


# A row of 900 bytes costs 7,217 units, one of a byte 25, a page takes rows that begin on 58,279 of them: with these numbers
# the rows end 3,604 units (57, 781) into a page, so the last row begins there or, when it is a long one, on the page before.
@pytest.mark.parametrize("longs,shorts", [(2000, 3243), (8, 24), (40, 2471)])
def test_last_row_on_either_page(pkg, ctx, oracle, longs, shorts):
    rng = np.random.default_rng(longs)
    words = ["y" * 900] * longs + ["z"] * shorts
    run(pkg, ctx, oracle, names(pkg, [words[i] for i in rng.permutation(len(words))], longs), f"{longs} {shorts}", 40)


@pytest.mark.parametrize("rows,longs", [(3000, 1), (6000, 7), (20_000, 40)])
def test_strings_of_several_pages(pkg, ctx, oracle, rows, longs):
    rng = np.random.default_rng(rows)
    words = ["x" * int(rng.integers(0, 60)) + str(i) for i in range(rows)]
    for i in rng.choice(rows, longs, replace=False):
        words[i] = "long" * int(rng.integers(2100, 6000))
    run(pkg, ctx, oracle, names(pkg, words, rows), f"{rows} {longs}", 12)
