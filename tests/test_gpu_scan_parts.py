"""The direct scan's blocks share a page where pages are few (eight, four, two blocks a page, one from 445 pages on, on 148
SMs): against the oracle on both sides of each line, alone and with the fused unique-key stages."""
import pytest

from test_gpu_scan_forms import check, star

pytestmark = pytest.mark.gpu


# 1,984 INT32 or 1,007 INT64 rows a page; the last page holds a lone row, or is full.
@pytest.mark.parametrize("pages", [111, 112, 222, 223, 444, 445])
@pytest.mark.parametrize("dims", [[400], [400, 90]])
@pytest.mark.parametrize("wide", [False, True])
def test_blocks_a_page(pkg, ctx, oracle, pages, dims, wide):
    fact = (1007 if wide else 1984) * pages - (0 if pages % 2 else (1007 if wide else 1984) - 1)
    check(pkg, ctx, oracle, star(pkg, pages, fact, dims, 0.3, 0.0, wide), f"pages {pages} dims {dims} wide {wide}")
