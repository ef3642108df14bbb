"""Keys that repeat many times on the build side: buckets a lane walks, buckets the warp walks (more than 32 entries in a
probe, more than 8 in the table's flags) and matches beyond a block's shared memory, against the oracle."""
import numpy as np
import pytest

from test_gpu_scan_forms import check, column

pytestmark = pytest.mark.gpu


# The hottest key's copies, on both sides of a lane's 8 and 32 entries, a warp's steps of 64, the flags' 256.
@pytest.mark.parametrize("copies", [7, 8, 9, 31, 32, 33, 95, 96, 97, 255, 257, 5000])
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("fed", [False, True])
def test_hot_keys(pkg, ctx, oracle, copies, wide, fed):
    rng = np.random.default_rng(copies)
    kt, kn = (pkg.INT64, np.int64) if wide else (pkg.INT32, np.int32)
    # Build side: key 0 `copies` times, key 1 half as often, 200 keys once; probe side: 40 hits on the hot keys among others.
    build = np.concatenate([np.zeros(copies), np.ones(copies // 2), np.arange(2, 202)]).astype(kn)
    rng.shuffle(build)
    probe = np.concatenate([np.repeat([0, 1], 20), rng.integers(2, 400, 3000)]).astype(kn)
    rng.shuffle(probe)
    p = pkg.Plan()
    a = p.new_input(pkg.ColumnarTable(len(probe), [column(pkg, kt, probe),
                                                   column(pkg, pkg.INT32, np.arange(len(probe), dtype=np.int32))]))
    left = p.new_scan_node(a, [(0, kt), (1, pkg.INT32)])
    b = p.new_input(pkg.ColumnarTable(len(build), [
        column(pkg, kt, build), column(pkg, pkg.INT32, np.arange(len(build), dtype=np.int32)),
        column(pkg, pkg.INT32, rng.integers(0, 50, len(build), dtype=np.int32))]))
    right = p.new_scan_node(b, [(0, kt), (1, pkg.INT32), (2, pkg.INT32)])
    if fed:  # the build's rows come through a probe of their own
        c = p.new_input(pkg.ColumnarTable(60, [column(pkg, pkg.INT32, np.arange(60, dtype=np.int32))]))
        right = p.new_join_node(False, right, p.new_scan_node(c, [(0, pkg.INT32)]), 2, 0, [(0, kt), (1, pkg.INT32),
                                                                                          (2, pkg.INT32)])
    p.root = p.new_join_node(False, left, right, 0, 0, [(1, pkg.INT32), (3, pkg.INT32), (4, pkg.INT32)])
    check(pkg, ctx, oracle, pkg.CPlan(p), f"copies {copies} wide {wide} fed {fed}")
