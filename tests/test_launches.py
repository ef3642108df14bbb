"""Host side of kernel launches, on the CPU: shared-memory attributes are kept for each device, a refused launch is
reported to the caller, also out of a capture."""
import glob
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "contest-sigmod2025_b200", "csrc")
CUDA = os.environ.get("CUDA", "/usr/local/cuda")


def _run(tmp_path, name, *sources):
    exe = str(tmp_path / name)
    subprocess.run(["g++", "-std=c++20", "-O1", "-pthread", "-I", CSRC, "-I", os.path.join(CUDA, "include"), "-o", exe,
                    os.path.join(HERE, "cpp", name + ".cpp"), *(os.path.join(CSRC, s) for s in sources)], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


def test_shared_memory_attribute_is_set_on_every_device(tmp_path):
    _run(tmp_path, "smem_attribute")
    for path in glob.glob(os.path.join(CSRC, "*.cu")):  # no launcher keeps its own once-flag
        assert "cudaFuncSetAttribute" not in open(path).read(), path


def test_refused_launch_is_reported(tmp_path):
    _run(tmp_path, "launch_status")


def test_an_exception_ends_the_capture(tmp_path):
    _run(tmp_path, "capture_exception", "graphs.cpp")
