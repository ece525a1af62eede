"""Where a plan's inputs wait for their step (csrc/cuda/step_inputs.hpp), in random sequences of setting, staging, accepting,
submitting and profiling: a step reads the plan's values and never a batch that no step of the run has accepted, the run keeps
its own values, and no slot is written that a step in flight reads."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    program = str(tmp_path_factory.mktemp("step_inputs") / "check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=address,undefined", "-I" + os.path.join(HERE, "..", "modelspec_b200", "csrc", "cuda"),
                    os.path.join(HERE, "host", "step_inputs_check.cpp"), "-o", program], check=True)
    return program


@pytest.mark.parametrize("seed", range(20))
def test_random_sequences(check, seed):
    ran = subprocess.run([check, str(seed)], capture_output=True, text=True, timeout=60)
    assert ran.returncode == 0, ran.stderr
    assert ran.stdout == "ok\n"
