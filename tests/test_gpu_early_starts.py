"""Kernels of a captured step that start while the ones before them end (MSX_FUSE bit 128), at sizes whose kernels run in several
waves and release the next one from the middle of their work: every loss, the state, a held-out evaluation and a prediction have
the bits that they have with every edge of the graph left as captured."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def results(mask):
    env = dict(os.environ, MSX_FUSE=mask, PYTHONPATH=os.pathsep.join([os.path.dirname(HERE), HERE, os.environ.get("PYTHONPATH", "")]))
    done = subprocess.run([sys.executable, os.path.join(HERE, "early_start_worker.py")], env=env, capture_output=True, text=True, timeout=900)
    assert done.returncode == 0, done.stderr[-2000:]
    return json.loads(done.stdout.strip().splitlines()[-1])


def test_the_bits_of_a_step_do_not_depend_on_when_its_kernels_start():
    late, early = results("127"), results("255")
    assert len(late) == 12 and late.keys() == early.keys()
    for case in late:
        assert late[case] == early[case], case
