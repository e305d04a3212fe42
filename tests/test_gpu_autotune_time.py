"""What the autotuner times are the steps, and not the capture of their graphs."""
import time

import pytest

from cuteflow_gb300 import cases

pytestmark = pytest.mark.gpu


def test_a_trials_time_is_that_of_its_steps(gpu_lib):
    """20 steps of 1,408 triangles take ~400 us; beside them an event pair sees one launch (below 10 us, 3 %).
    With 3 % for the timer on either side: within 10 % of a long run in the setting that was picked."""
    from cuteflow_gb300 import Solver
    c = cases.channel(44, 16, lx=440.0, ly=160.0, iflux=2, inlet=2)
    with Solver(c) as s:
        s.set_state(c.U0)
        s.step(1000)
        ms = min(s.autotune(20)[2] for _ in range(3))
        s.step(1000)
        long = []
        for _ in range(3):
            t = time.perf_counter()
            s.step(1000)
            long.append(1e3 * (time.perf_counter() - t) / 1000)
    print(f"autotune {1e3 * ms:.2f} us, 1000 steps {1e3 * min(long):.2f} us per step")
    assert ms <= 1.10 * min(long)
