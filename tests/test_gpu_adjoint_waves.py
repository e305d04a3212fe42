"""The reverse edge kernel's two register budgets: a mesh on either side of each line between them has the
gradients it has as a member of a batch whose size takes the other one, bit for bit."""
import numpy as np
import pytest

from cuteflow_gb300 import cases

pytestmark = pytest.mark.gpu


# 455, 457, 608 and 610 tiles of 128 edges; a batch of two is beyond both lines
@pytest.mark.parametrize("ny", [193, 194, 258, 259])
def test_gradients_do_not_depend_on_the_register_budget(gpu_lib, ny):
    from cuteflow_gb300 import Batch, Solver
    from cuteflow_gb300.adjoint import Adjoint
    c = cases.circular_dam_break(100, ny, seed=ny, iflux=1)
    gauges = np.array([5, c.nelt // 2, c.nelt - 1], np.int32)
    with Solver(c) as s, Adjoint(s, 4, gauges) as adj:
        s.set_state(c.U0)
        eta, _ = adj.forward()
        w = np.linspace(-1.0, 1.0, eta.size).reshape(eta.shape)
        ws = 0.01 * np.ones((c.nelt, 3))
        gU, gn = adj.backward(w, ws)
    gm = np.repeat(np.array([0, 1], np.int32), 3)
    with Batch([c, c]) as b, Adjoint(b, 4, np.tile(gauges, 2), gauge_member=gm) as adj:
        for m in (0, 1):
            b.set_state(m, c.U0)
        adj.forward()
        gU2, gn2 = adj.backward(np.tile(w, (1, 2)), np.tile(ws, (2, 1)))
    for m in (0, 1):
        assert np.array_equal(gU2[m * c.nelt:(m + 1) * c.nelt], gU)
        assert np.array_equal(gn2[m * c.nelt:(m + 1) * c.nelt], gn)
