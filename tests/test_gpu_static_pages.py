"""bj_join_count_static over more probe pages than blocks run together: counts at the blocks' turns, and what many pages
against a small table take."""
import numpy as np
import pytest

from test_gpu_static_sizes import _pages
from test_zz_no_alloc import ERR_COUNT, count_static

pytestmark = pytest.mark.gpu

BLOCKS = 148 * 6
FULL = 1984  # rows of a full page


# A block's first turn, its second, a third for some.
@pytest.mark.parametrize("pages", [BLOCKS - 1, BLOCKS, BLOCKS + 1, 2 * BLOCKS, 2 * BLOCKS + 1])
@pytest.mark.parametrize("build", [0, 700])
def test_turns(pkg, pages, build):
    import torch

    rng = np.random.default_rng(pages)
    b = rng.integers(0, 500, build)
    p = rng.integers(0, 1000, (pages - 1) * FULL + 1)
    db, nb = _pages(pkg, b, np.ones(build, bool))
    dp, npp = _pages(pkg, p, np.ones(len(p), bool))
    assert npp == pages
    want = int(np.bincount(b, minlength=1000)[p].sum()) if build else 0
    out = torch.full((1,), -1, dtype=torch.int64, device="cuda")
    assert count_static(pkg, db, nb, build, dp, npp, out) == (0, want)
    dp.view(torch.int16)[(pages - 1) * 4096] = 0  # the last page: one value, no rows
    assert count_static(pkg, db, nb, build, dp, npp, out) == (0, ERR_COUNT)


def test_many_pages_against_a_small_table(pkg):
    """What 16M rows against 5,000 keys take, by what they take against 262,144, whose slots miss L1."""
    import torch

    rng = np.random.default_rng(1)
    dp, npp = _pages(pkg, rng.integers(0, 10_000, 16_000_000), np.ones(16_000_000, bool))
    out = torch.zeros(1, dtype=torch.int64, device="cuda")
    builds = [(n, *_pages(pkg, rng.integers(0, 10_000 if n == 5000 else 1 << 30, n), np.ones(n, bool))) for n in (5000, 262_144)]
    dq, nq = _pages(pkg, rng.integers(0, 1 << 30, 16_000_000), np.ones(16_000_000, bool))
    best = [1e9, 1e9]
    for _ in range(25):
        for k, (n, db, nb) in enumerate(builds):
            probe, pages = (dp, npp) if k == 0 else (dq, nq)
            begin, end = torch.cuda.Event(True), torch.cuda.Event(True)
            begin.record()
            # (Not count_static: it waits for the count before the end is recorded.)
            assert pkg.lib().bj_join_count_static(db.data_ptr(), nb, n, probe.data_ptr(), pages, out.data_ptr(), None) == 0
            end.record()
            torch.cuda.synchronize()
            best[k] = min(best[k], begin.elapsed_time(end) * 1e3)
    # 54 to 92 us; with a block a page, each ending in its own atomics, 87 to 109.
    assert best[0] < 0.70 * best[1], best
