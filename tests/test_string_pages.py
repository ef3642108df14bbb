"""The pages of a VARCHAR result column, planned for rows in any order, on the CPU."""
from test_launches import _run


def test_pages_in_any_order(tmp_path):
    _run(tmp_path, "string_pages")
