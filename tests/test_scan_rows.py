"""The staged scan's search for a value's row in a page with NULLs, compiled for the CPU."""
from test_launches import _run


def test_row_of_a_value(tmp_path):
    _run(tmp_path, "page_rows")
