"""A build that turns out empty ends its query at the next pipeline that probes it, also where its size is not read back."""
import ctypes

import numpy as np
import pytest

import oracle_lib
from test_gpu_scan_forms import column

pytestmark = pytest.mark.gpu


def chain(pkg, hits):
    """fact -> c -> b -> u, `hits` rows of b referring to a key of u."""
    rng = np.random.default_rng(hits)
    i32 = pkg.INT32
    ints = lambda v: column(pkg, i32, np.asarray(v, np.int32))  # noqa: E731
    nf, nc, nb, nu = 200_000, 30_000, 20_000, 500
    to_u = 1000 + rng.integers(0, 10_000, nb)
    to_u[:hits] = 7
    to_b = rng.integers(0, nb, nc)
    to_b[:50] = 0
    p = pkg.Plan()
    p.new_input(pkg.ColumnarTable(nf, [ints(rng.integers(0, nc, nf)), ints(np.arange(nf))]))
    p.new_input(pkg.ColumnarTable(nc, [ints(rng.permutation(nc)), ints(to_b)]))
    p.new_input(pkg.ColumnarTable(nb, [ints(np.arange(nb)), ints(to_u)]))
    p.new_input(pkg.ColumnarTable(nu, [ints(rng.permutation(nu))]))
    left = p.new_scan_node(0, [(0, i32), (1, i32)])
    left = p.new_join_node(False, left, p.new_scan_node(1, [(0, i32), (1, i32)]), 0, 0, [(1, i32), (3, i32)])
    left = p.new_join_node(False, left, p.new_scan_node(2, [(0, i32), (1, i32)]), 1, 0, [(0, i32), (3, i32)])
    p.root = p.new_join_node(False, left, p.new_scan_node(3, [(0, i32)]), 1, 0, [(0, i32)])
    return pkg.CPlan(p)


@pytest.mark.parametrize("hits", [0, 1, 300])
def test_empty_build_ends_the_query(pkg, oracle, hits):
    cp = chain(pkg, hits)
    want = oracle.execute(cp.ref())
    plan = cp.struct
    for graphs in (False, True):
        ctx = pkg.Context(0)
        try:
            ctx.set_graphs(graphs)
            res = [ctx.upload(plan.inputs[i]) for i in range(plan.num_inputs)]
            for run in range(4):
                with ctx.execute_resident(cp, res) as r:
                    got, keep = r.table_struct()
                    n = oracle_lib.assert_same_rows(oracle, ctypes.byref(got), want.view(), f"{hits} {graphs} {run}")
                    assert (n > 0) == (hits > 0)
                    assert r.stats().pipelines == (4 if hits else 3)  # u, b, c (which finds b empty), and the fact
            for x in res:
                x.free()
        finally:
            ctx.close()
