"""The estimator's row stage under several threads, on the CPU, over a runtime of the test's own."""
from test_launches import _run


def test_uploads_of_many_threads(tmp_path):
    _run(tmp_path, "row_stage")
