"""The recording forward in every launch shape: the dt and gauge records and the gradients are the same bits,
on meshes whose last block is partly empty (and the gauges' block comes after it)."""
import numpy as np
import pytest

from cuteflow_gb300 import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("iflux", [1, 2, 3])
@pytest.mark.parametrize("size", [(3, 2), (23, 11), (60, 41)])
def test_records_do_not_depend_on_the_shape(gpu_lib, iflux, size):
    from cuteflow_gb300 import Solver
    from cuteflow_gb300.adjoint import Adjoint
    c = cases.circular_dam_break(*size, seed=5, iflux=iflux)
    gauges = np.array([0, c.nelt // 2, c.nelt - 1], np.int32)
    ref = None
    for shape in (None, (64, 1, 128), (64, 2, 128), (128, 1, 256), (128, 2, 128), (256, 1, 128), (256, 2, 256)):
        with Solver(c) as s:
            if shape:
                s.set_launch_shape(*shape)
            with Adjoint(s, 5, gauges) as adj:
                s.set_state(c.U0)
                eta, U = adj.forward()
                g = adj.backward(np.ones_like(eta), 0.1 * np.ones((c.nelt, 3)))
                got = [eta, U, *adj.dt_history(), *g]
        if ref is None:
            ref = got
        assert all(np.array_equal(a, b) for a, b in zip(ref, got)), shape
