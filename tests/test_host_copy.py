"""The staged download (csrc/cuda/host_copy.hpp) against host memory in the place of the device's: a
process that may start no more threads, or only some, gets its bytes all the same, and the first error
of any thread is the result."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    program = str(tmp_path_factory.mktemp("host_copy") / "check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + os.path.join(HERE, "host"), "-I" + os.path.join(HERE, "..", "modelspec_b200", "csrc", "cuda"),
                    os.path.join(HERE, "host", "host_copy_check.cpp"), "-o", program, "-pthread", "-ldl"], check=True)
    return lambda threads, fails, registers=1: subprocess.run([program, str(threads), str(fails), str(registers)], capture_output=True, text=True, timeout=60)


@pytest.mark.parametrize("threads", [0, 1, 3, 7, 1000])
@pytest.mark.parametrize("registers", [0, 1])
def test_a_download_needs_no_thread(check, threads, registers):
    ran = check(threads, -1, registers)
    assert ran.returncode == 0, ran.stderr
    assert ran.stdout == "0 whole\n"


@pytest.mark.parametrize("threads", [0, 7])
@pytest.mark.parametrize("first", [0, 5, 20])
def test_the_first_error_is_the_result(check, threads, first):
    ran = check(threads, first)
    assert ran.returncode == 0, ran.stderr
    assert ran.stdout == "1 not whole\n"
