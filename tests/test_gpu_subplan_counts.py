"""Exact sub-plan counts against counts over flat arrays: shared passes (more
options and more totals than one pass takes, several roots), maps of sub-trees
several levels deep, NULL keys, counts past 2^64 - 1."""
import ctypes

import numpy as np
import pytest

from test_gpu_scan_forms import column

pytestmark = pytest.mark.gpu


def _tree(pkg, seed, edges, rows, wide, domain):
    """Tables t (rows[t] rows) with a column per edge end; edges (a, b) joined on values below `domain`. Scans in the
    order of a depth-first walk are the tables in order."""
    rng = np.random.default_rng(seed)
    kt = pkg.INT64 if wide else pkg.INT32
    cols = [[] for _ in rows]
    place = {}
    for e, (a, b) in enumerate(edges):
        for t in (a, b):
            place[e, t] = len(cols[t])
            v = rng.integers(0, domain, rows[t])
            v = np.where(rng.random(rows[t]) < 0.05, domain - 1, v)  # a heavy key
            ok = rng.random(rows[t]) >= 0.1
            cols[t].append((v.astype(np.int64) - 3, ok))
    p = pkg.Plan()
    for t, n in enumerate(rows):
        p.new_input(pkg.ColumnarTable(n, [
            column(pkg, kt, v if wide else v.astype(np.int32), ok.astype(np.uint8)) for v, ok in cols[t]]))
    at = {}
    left, width = None, 0
    for t in range(len(rows)):
        scan = p.new_scan_node(t, [(c, kt) for c in range(len(cols[t]))])
        if left is None:
            left = scan
        else:
            e = next(e for e, (a, b) in enumerate(edges) if b == t)
            k = len(cols[t])
            left = p.new_join_node(False, left, scan, at[e, edges[e][0]], place[e, t], [(i, kt) for i in range(width + k)])
        for e, (a, b) in enumerate(edges):
            if t in (a, b):
                at[e, t] = width + place[e, t]
        width += len(cols[t])
    p.root = left
    return pkg.CPlan(p), cols, place


def _count(cols, place, edges, mask):
    def weights(t, parent):
        w = [1] * len(cols[t][0][0])
        for e, (a, b) in enumerate(edges):
            if t not in (a, b) or e == parent:
                continue
            o = b if t == a else a
            if not mask >> o & 1:
                continue
            sums = {}
            for v, ok, x in zip(*cols[o][place[e, o]], weights(o, e)):
                if ok:
                    sums[int(v)] = sums.get(int(v), 0) + x
            w = [x * sums.get(int(v), 0) if ok else 0 for x, v, ok in zip(w, *cols[t][place[e, t]])]
        return w
    return sum(weights((mask & -mask).bit_length() - 1, None))


STAR = [(0, t) for t in range(1, 8)]                            # 127 sub-plans rooted at the centre: two passes
CHAIN = [(0, 1), (1, 2), (2, 3), (3, 4)]                        # maps of maps
BUSHY = [(0, 1), (1, 2), (0, 3), (3, 4), (3, 5), (0, 6)]        # more options at the root than one pass takes


@pytest.mark.parametrize("name", ["star", "chain", "bushy"])
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("rows", [1, 255, 700])
def test_counts(pkg, ctx, name, wide, rows):
    edges = {"star": STAR, "chain": CHAIN, "bushy": BUSHY}[name]
    sizes = [rows] + [max(1, rows // (2 + t % 3)) for t in range(1, 1 + max(b for _, b in edges))]
    cp, cols, place = _tree(pkg, rows, edges, sizes, wide, 40)
    res = [ctx.upload(cp.struct.inputs[i]) for i in range(len(sizes))]
    try:
        masks = pkg.subplans(cp)
        got = ctx.subplan_cards(cp, res, masks)
        for m, g in zip(masks, got):
            m = int(m)
            want = _count(cols, place, edges, m) if m & (m - 1) else sizes[m.bit_length() - 1]
            assert g == float(want), f"{name} {m:#x}: {g} != {want}"
    finally:
        for x in res:
            x.free()


def test_counts_past_64_bits_are_infinite(pkg, ctx):
    """One key everywhere: products of row counts, below and above 2^64."""
    rows = [3000] * 7
    edges = [(0, 1), (1, 2), (2, 3), (3, 4), (4, 5), (0, 6)]
    cp, _, _ = _tree(pkg, 1, edges, rows, False, 1)
    plan = cp.struct
    res = [ctx.upload(plan.inputs[i]) for i in range(7)]
    try:
        masks = pkg.subplans(cp)
        got = dict(zip((int(m) for m in masks), ctx.subplan_cards(cp, res, masks)))
        for m, g in got.items():
            n = bin(m).count("1")
            if n >= 7:
                assert np.isinf(g), f"{m:#x}: {g}"
            elif n <= 5:
                assert np.isfinite(g), f"{m:#x}: {g}"
    finally:
        for x in res:
            x.free()
