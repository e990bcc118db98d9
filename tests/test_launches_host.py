"""The launches the library's host code issues, without a GPU: its objects
linked with a stand-in CUDA runtime that writes launches down instead of
running them (tests/host/)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")
OBJECTS = ["kernels", "kernels_mixed", "capi", "ensemble", "checkpoint", "geometry", "peaks"]

pytestmark = pytest.mark.skipif(
    shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA, "bin", "nvcc")),
    reason="no compiler")


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    subprocess.run(["make", "-s", "-C", os.path.join(ROOT, "exocubed_b200", "csrc")], check=True)
    exe = str(tmp_path_factory.mktemp("host") / "launch_driver")
    cmd = ["g++", "-std=c++17", "-O1", "-g", "-Wall", f"-I{CUDA}/include",
           *[os.path.join(ROOT, "tests", "host", f) for f in ("launch_driver.cpp", "host_cuda.cpp")],
           *[os.path.join(ROOT, "_build", "csrc", o + ".o") for o in OBJECTS], "-pthread", "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    return exe


def _check(driver, what):
    r = subprocess.run([driver, what], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and f"{what}: ok" in r.stdout, r.stdout + r.stderr


def test_launches_of_a_column_solve_stay_together(driver):
    _check(driver, "pairs")


def test_a_wait_that_gave_up_is_the_implicit_call_s_error(driver):
    _check(driver, "timeout")


def test_column_hooks_take_the_deepest_columns(driver):
    _check(driver, "levels")


def test_the_mixed_solve_leaves_its_l1(driver):
    _check(driver, "fused_smem")
