"""Exact sub-plan counts around 2^64: sums of an inner table's map and products that pass it are infinite in every sub-plan
that joins them, and in no other. Against counts in Python integers."""
import numpy as np
import pytest

from test_gpu_scan_forms import column
from test_gpu_subplan_counts import _count

pytestmark = pytest.mark.gpu


def plan(pkg, tables, edges):
    """tables[t]: {edge: INT64 keys of table t on that edge}; edges (a, b), each table's edge to an earlier one first."""
    p = pkg.Plan()
    cols, place = [], {}
    for t, own in enumerate(tables):
        cols.append([])
        for e, v in own.items():
            place[e, t] = len(cols[t])
            cols[t].append((np.asarray(v, np.int64), np.ones(len(v), bool)))
        p.new_input(pkg.ColumnarTable(len(cols[t][0][0]), [column(pkg, pkg.INT64, v) for v, _ in cols[t]]))
    at, left, width = {}, None, 0
    for t in range(len(tables)):
        scan = p.new_scan_node(t, [(c, pkg.INT64) for c in range(len(cols[t]))])
        if left is None:
            left = scan
        else:
            e = next(e for e, (_, b) in enumerate(edges) if b == t)
            left = p.new_join_node(False, left, scan, at[e, edges[e][0]], place[e, t],
                                   [(i, pkg.INT64) for i in range(width + len(cols[t]))])
        for e, (a, b) in enumerate(edges):
            if t in (a, b):
                at[e, t] = width + place[e, t]
        width += len(cols[t])
    p.root = left
    return pkg.CPlan(p), cols, place


def check(pkg, ctx, tables, edges):
    cp, cols, place = plan(pkg, tables, edges)
    res = [ctx.upload(cp.struct.inputs[i]) for i in range(len(tables))]
    try:
        masks = pkg.subplans(cp)
        got = dict(zip((int(m) for m in masks), ctx.subplan_cards(cp, res, masks)))
        infinite = 0
        for m, g in got.items():
            n = _count(cols, place, edges, m) if m & (m - 1) else len(cols[m.bit_length() - 1][0][0])
            want = float("inf") if n >= 1 << 64 else float(n)
            assert g == want, f"{m:#x}: {g} != {want} ({n})"
            infinite += n >= 1 << 64
        # Each sub-plan alone too, in a pass of its own.
        for m in got:
            assert ctx.subplan_cards(cp, res, np.array([m], masks.dtype))[0] == got[m], f"{m:#x} alone"
        return infinite
    finally:
        for x in res:
            x.free()


CHAIN = [(t, t + 1) for t in range(6)]


def chain(k, rows):
    return [{e: np.full(rows[t], k) for e, edge in enumerate(CHAIN) if t in edge} for t in range(7)]


# A map's sum is 15, 16 and 17 times 2^60: 16 wraps to 0, as if the key were not there. The key -1 has a slot of its own.
@pytest.mark.parametrize("k", [1, -1])
@pytest.mark.parametrize("n", [15, 16, 17])
@pytest.mark.parametrize("root", [1, 300])
def test_sum_of_a_map(pkg, ctx, k, n, root):
    infinite = check(pkg, ctx, chain(k, [root, n] + [4096] * 5), CHAIN)
    assert infinite == (2 if n >= 16 else root * n >= 16)  # tables 1 to 6, and all seven


def test_deep_chain_of_one_key(pkg, ctx):
    """Every map past the fifth level sums past 2^64."""
    assert check(pkg, ctx, chain(7, [3000] * 7), CHAIN) == 3  # seven tables, and the two chains of six


def test_sum_that_nothing_joins(pkg, ctx):
    """Key 9's sum passes 2^64, key 5's does not, and the root has only key 5."""
    tables = chain(1, [2] + [3000] * 6)
    tables[0][0] = np.array([5, 5])
    tables[1][0] = np.where(np.arange(3000) < 1, 5, 9)
    assert check(pkg, ctx, tables, CHAIN) == 1  # tables 1 to 6 by themselves


def test_product_that_nothing_joins(pkg, ctx):
    """Table 1 multiplies two children of 2^36 each: past 2^64 in rows that the root does not join, or joins."""
    edges = [(0, 1), (1, 2), (2, 3), (3, 4), (1, 5), (5, 6), (6, 7)]
    for root in (5, 9):
        tables = [{e: np.full(4096, 1) for e, edge in enumerate(edges) if t in edge} for t in range(8)]
        tables[0][0] = np.array([root, root])
        tables[1] = {0: np.array([5, 9]), 1: np.array([1, 1]), 4: np.array([2, 1])}  # key 5 finds nothing on edge 4
        assert check(pkg, ctx, tables, edges) == (2 if root == 9 else 1)
