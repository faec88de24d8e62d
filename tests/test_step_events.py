"""A step's time is read from its events only after the closing event has been
waited for: the wait for a step's result (a number in pinned memory) does not
promise that the event reads as complete, and an early read turns a finished
step into an error.  Checked in the sources (it cannot be provoked), and on the
GPU over many short steps."""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "finess_b200", "csrc")


@pytest.mark.parametrize("name", ["finess_b200.cu", "fin_mhd.cu", "fin_batch.cu"])
def test_elapsed_times_follow_a_wait(name):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    reads = list(re.finditer(r"cudaEventElapsedTime\(&\w+, ([\w>-]*)ev0, \1ev1\)", text))
    assert reads
    for m in reads:
        body = text[text.rfind("\n}\n", 0, m.start()):m.start()]   # the function up to the read
        assert f"cudaEventSynchronize({m.group(1)}ev1)" in body, (name, text.count("\n", 0, m.start()) + 1)


@pytest.mark.gpu
def test_many_short_mhd_steps():
    from finess_b200 import problems as P
    from finess_b200.mhd import MhdSolver
    p = P.orszag_tang_params(n=16)
    q, aux = P.mhd_random_state(p, np.random.default_rng(5))
    with MhdSolver(p) as s:
        s.set_state(q, aux)
        for _ in range(2000):
            s.step_fixed(1e-7)
