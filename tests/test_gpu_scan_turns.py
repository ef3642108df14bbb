"""The direct scan's blocks with more rows than one turn takes (3,072): INT32 and INT64 key columns whose NULLs put so many
rows into a page, one block a page and several, with a filter and without, turns that match nothing before turns that do.
Before every run the estimator's products leave their operands in shared memory, so that a word a kernel did not write
itself is not zero by luck. Against the oracle."""
import ctypes

import numpy as np
import pytest

import oracle_lib
from test_gpu_scan_forms import column

pytestmark = pytest.mark.gpu

TURN = 3072


@pytest.fixture(scope="module")
def dirty(pkg):
    est = pkg.Estimator(0, seed=1)
    x = np.random.default_rng(1).uniform(0.5, 1.0, (4096, pkg.EST_FEATURES)).astype(np.float32)
    return lambda: est.predict(x)


def paged(pkg, wide, pages):
    """A column of the given pages, each (values, valid)."""
    w = 8 if wide else 4
    out = bytearray()
    for values, valid in pages:
        dense, bits = values[valid], np.packbits(valid, bitorder="little").tobytes()
        pg = bytearray(8192)
        pg[0:4] = np.array([len(valid), len(dense)], np.uint16).tobytes()
        pg[w:w + w * len(dense)] = dense.astype(np.int64 if wide else np.int32).tobytes()
        assert w + w * len(dense) + len(bits) <= 8192
        pg[8192 - len(bits):] = bits
        out += pg
    return pkg.Column(pkg.INT64 if wide else pkg.INT32, bytes(out))


def lookup(pkg, rng, rows, key, wide, present, dim):
    """fact(key, id) joined with a table of `dim` keys, `present` among them."""
    kt = pkg.INT64 if wide else pkg.INT32
    own = present if len(present) >= dim else np.concatenate([present, np.arange(dim - len(present)) * 2 + (1 << 29)])
    p = pkg.Plan()
    p.new_input(pkg.ColumnarTable(rows, [key, column(pkg, pkg.INT32, np.arange(rows, dtype=np.int32))]))
    p.new_input(pkg.ColumnarTable(len(own), [
        column(pkg, kt, rng.permutation(own).astype(np.int64 if wide else np.int32)),
        column(pkg, pkg.INT32, rng.integers(0, 1 << 30, len(own), dtype=np.int32))]))
    a = p.new_scan_node(0, [(0, kt), (1, pkg.INT32)])
    b = p.new_scan_node(1, [(0, kt), (1, pkg.INT32)])
    p.root = p.new_join_node(False, a, b, 0, 0, [(0, kt), (1, pkg.INT32), (3, pkg.INT32)])
    return pkg.CPlan(p)


def check(pkg, ctx, oracle, dirty, cp, label):
    want = oracle.execute(cp.ref())
    plan = cp.struct
    res = [ctx.upload(plan.inputs[i]) for i in range(plan.num_inputs)]
    try:
        for run in range(4):  # recorded, captured, replayed twice
            dirty()
            with ctx.execute_resident(cp, res) as r:
                got, keep = r.table_struct()
                assert oracle_lib.assert_same_rows(oracle, ctypes.byref(got), want.view(), f"{label} run {run}") > 0
    finally:
        for x in res:
            x.free()


# dim 3,000: INT32 tables have a filter; 140,000: none has (nor has an INT64 one). One block a page from 445 pages on, eight
# at 60; a filtered scan takes this form up to 512 pages.
@pytest.mark.parametrize("wide,nulls,pages", [(False, 0.4, 446), (False, 0.4, 600), (False, 0.7, 460), (False, 0.97, 60),
                                              (True, 0.7, 450), (True, 0.9, 223), (True, 0.9, 520)])
@pytest.mark.parametrize("dim", [3000, 140_000])
@pytest.mark.parametrize("match", [0.001, 0.3])
def test_sparse_matches(pkg, ctx, oracle, dirty, wide, nulls, pages, dim, match):
    rng = np.random.default_rng(pages)
    w = 8 if wide else 4
    rows = int(pages * (8192 - w) / (w * (1 - nulls) + 0.125))
    hit = rng.random(rows) < match
    fk = np.where(hit, rng.integers(0, 1000, rows) * 2, rng.integers(0, 1 << 28, rows) * 2 + 1)
    if wide:
        fk = fk | (5 << 33)
    present = np.arange(1000, dtype=np.int64) * 2 | (5 << 33 if wide else 0)
    key = column(pkg, pkg.INT64 if wide else pkg.INT32, fk.astype(np.int64 if wide else np.int32),
                 (rng.random(rows) >= nulls).astype(np.uint8))
    check(pkg, ctx, oracle, dirty, lookup(pkg, rng, rows, key, wide, present, dim), f"{wide} {nulls} {pages} {dim} {match}")


# Pages that begin with a turn (or two) of NULLs, or of keys that miss, before the rows that match.
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("before", [TURN, 2 * TURN + 64])
@pytest.mark.parametrize("npages", [112, 450])
@pytest.mark.parametrize("dim", [3000, 140_000])
def test_first_turn_without_a_match(pkg, ctx, oracle, dirty, wide, before, npages, dim):
    rng = np.random.default_rng(before + npages)
    present = np.arange(1000, dtype=np.int64) * 2
    pages, rows = [], 0
    for p in range(npages):
        n = before + 300 + p % 7
        valid = np.zeros(n, bool)
        valid[before:] = rng.random(n - before) < 0.9
        values = present[rng.integers(0, 1000, n)]
        if p % 3 == 0:  # some keys before, none of them there
            valid[:before] = rng.random(before) < 0.05
            values[:before] = 2 * values[:before] + (1 << 28) + 1
        pages.append((values, valid))
        rows += n
    check(pkg, ctx, oracle, dirty, lookup(pkg, rng, rows, paged(pkg, wide, pages), wide, present, dim),
          f"{wide} {before} {npages} {dim}")
