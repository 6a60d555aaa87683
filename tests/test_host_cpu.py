"""Host code of the library that no GPU is needed for, built against stand-ins for the CUDA runtime
(tests/host): what it does when an allocation, a stream or a copy cannot be had."""
import os
import subprocess

import pytest

from tests.helpers import ROOT

CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")
CSRC = os.path.join(ROOT, "pcaone_b200", "csrc")


def program(tmp_path, test, *sources):
    exe = str(tmp_path / test)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-Wall", "-pthread", f"-I{CUDA}/include", "-o", exe,
                           os.path.join(ROOT, "tests", "host", test + ".cpp"), "-x", "c++",
                           *(os.path.join(CSRC, s) for s in sources)])
    return exe


def run(exe, *args):
    r = subprocess.run([exe, *args], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr


def test_buffers_survive_failed_allocations(tmp_path):
    run(program(tmp_path, "buffers_test", "buffers.cu"))


def test_row_split_of_the_tall_passes(tmp_path):
    """Every row count and cluster limit, down to a device that holds one cluster (or none beside the
    one set aside for the signs): the clusters cover the rows and keep to the limit."""
    exe = str(tmp_path / "tall")
    subprocess.check_call([f"{CUDA}/bin/nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-o", exe,
                           os.path.join(ROOT, "tests", "host", "tall_test.cu")])
    run(exe)


@pytest.fixture(scope="module")
def xfer(tmp_path_factory):
    return program(tmp_path_factory.mktemp("xfer"), "xfer_test", "xfer.cu")


@pytest.mark.parametrize("case", ["cold", "large", "no_slots", "pinned", "failed", "at_once"])
def test_large_host_copies(xfer, case):
    run(xfer, case)
