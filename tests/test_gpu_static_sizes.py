"""bj_join_count_static at the sizes where its table grows (twice the build
rows, powers of two), where a page's quarters and a thread's values end, and
without probe pages; counts against numpy."""
import numpy as np
import pytest

from test_gpu_scan_forms import column
from test_zz_no_alloc import ERR_COUNT, count_static

pytestmark = pytest.mark.gpu


def _pages(pkg, values, valid):
    import torch

    c = column(pkg, pkg.INT32, values.astype(np.int32), valid.astype(np.uint8))
    return torch.frombuffer(bytearray(c.data or b"\0" * 8192), dtype=torch.uint8).to("cuda"), c.num_pages


@pytest.mark.parametrize("build", [0, 1, 511, 512, 513, 1024, 1025, 131_072, 131_073, 262_144])
@pytest.mark.parametrize("probe", [0, 1, 512, 513, 1985, 70_001])
@pytest.mark.parametrize("distinct", [1, 1000, 1 << 30])
def test_counts(pkg, build, probe, distinct):
    import torch

    rng = np.random.default_rng(build + probe)
    b, p = rng.integers(-3, distinct, build), rng.integers(-3, distinct, probe)
    if build and probe:
        p[::2] = rng.choice(b, len(p[::2]))
    vb, vp = rng.random(build) >= 0.1, rng.random(probe) >= 0.1
    db, nb = _pages(pkg, b, vb)
    dp, npp = _pages(pkg, p, vp)
    keys, counts = np.unique(b[vb], return_counts=True)
    at = np.searchsorted(keys, p[vp])
    hit = (at < len(keys)) & (keys[np.minimum(at, max(len(keys) - 1, 0))] == p[vp]) if len(keys) else np.zeros(0, bool)
    want = int(counts[at[hit]].sum()) if len(keys) else 0
    out = torch.full((1,), -1, dtype=torch.int64, device="cuda")
    assert count_static(pkg, db, nb, build, dp, npp, out) == (0, want)
    if vb.sum():  # one row fewer than the pages hold
        assert count_static(pkg, db, nb, int(vb.sum()) - 1, dp, npp, out) == (0, ERR_COUNT)
