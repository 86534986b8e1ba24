"""The block cache behind every device allocation (gpr_cache.cc), on the host against a
CUDA runtime that only keeps books (cache_driver.cc): when it waits for the GPU, for
which device, and what it does where that wait is refused."""
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("cache") / "cache_driver")
    csrc = os.path.join(ROOT, "gardenia_ocl_b200", "csrc")
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O1", "-pthread", "-o", out,
                    os.path.join(ROOT, "tests", "cache_driver.cc"),
                    os.path.join(csrc, "gpr_cache.cc"), "-I", os.path.join(ROOT, "include"),
                    "-I", csrc, "-I", os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"),
                                                   "include")], check=True)

    def run(case):
        p = subprocess.run([out, case], capture_output=True, text=True, timeout=60)
        assert p.returncode == 0, p.stderr
        return p.stdout
    return run


def test_one_wait_for_all_blocks_freed_before(driver):
    assert driver("waits") == "ok\n"


def test_a_refused_wait_hands_out_nothing(driver):
    assert driver("refused") == "ok\n"


def test_other_threads_go_on_while_one_waits(driver):
    assert driver("threads") == "ok\n"


def test_gpr_free_waits_for_the_device_of_the_block(driver):
    assert driver("free") == "ok\n"
