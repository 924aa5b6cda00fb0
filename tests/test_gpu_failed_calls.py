"""A CUDA call that fails is reported once: it leaves no error for a later call's launch check and no
stream in capture (failed_calls.cu, compiled here)."""
import os
import subprocess

import pytest

import build as pkg_build

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    try:
        nvcc = pkg_build._nvcc()
    except RuntimeError:
        pytest.skip("nvcc not found")
    out = str(tmp_path_factory.mktemp("failed_calls") / "failed_calls")
    subprocess.run([nvcc, *pkg_build.ARCH, "-O1", "-std=c++17", "--expt-relaxed-constexpr",
                    "-I", os.path.join(pkg_build.REPO, "include"), "-I", pkg_build.CSRC,
                    os.path.join(HERE, "failed_calls.cu"), "-o", out], check=True)
    return out


def _run(program, what):
    r = subprocess.run([program, what], capture_output=True, text=True, timeout=120)
    assert (r.returncode, r.stdout.strip()) == (0, "ok"), r.stdout + r.stderr


def test_error_is_reported_once(program):
    _run(program, "allocation")


def test_capture_is_ended(program):
    _run(program, "capture")
