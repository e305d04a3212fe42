"""A trial of the autotuner that fails leaves the context as it was."""
import numpy as np
import pytest

from cuteflow_gb300 import cases

pytestmark = pytest.mark.gpu


def test_a_failed_autotune_restores_the_state(gpu_lib, oracle):
    from cuteflow_gb300 import Solver
    from cuteflow_gb300.solver import CFError
    c = cases.circular_dam_break(30, 20, seed=1, iflux=1)
    c.params.update(is_dt_constant=1, constant_dt=20000.0)   # out of the range that the second step tests
    with Solver(c) as s:
        s.set_state(c.U0)
        tuning, shape = s.tuning(), s.launch_shape()
        with pytest.raises(CFError, match="dt left the range"):
            s.autotune(4)
        assert (s.tuning(), s.launch_shape()) == (tuning, shape)
        info = s.info()
        assert info.status == 0 and info.steps == 0 and info.t == 0.0
        assert np.array_equal(s.get_state(), c.U0)
        assert s.step(1, check=False).steps == 1
        assert np.array_equal(s.get_state(), oracle.run(c, 1, check=False)["U"])
