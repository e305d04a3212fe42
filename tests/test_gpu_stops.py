"""Members that stop in the middle of a call, each at its own step, in every launch shape: the sides of
their edges leave or stay as whole warps, and the state is the one of the member alone."""
import numpy as np
import pytest

from cuteflow_gb300 import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(64, 1, 128), (64, 2, 128), (128, 1, 256), (128, 2, 128), (256, 1, 128), (256, 2, 256)])
@pytest.mark.parametrize("iflux", [1, 3])
def test_members_stop_at_their_own_step(gpu_lib, oracle, iflux, shape):
    from cuteflow_gb300 import Batch
    cs = [cases.circular_dam_break(nx, ny, seed=nx, iflux=iflux) for nx, ny in ((9, 7), (14, 11), (23, 17))]
    ts = 0.9 * oracle.run(cs[0], 40)["t"]
    with Batch(cs) as b:
        b.set_launch_shape(*shape)
        for m, c in enumerate(cs):
            b.set_state(m, c.U0)
        infos = b.run(ts, max_steps=400)
        steps = [i.steps for i in infos]
        assert len(set(steps)) == 3 and max(steps) < 400
        for m, c in enumerate(cs):
            ref = oracle.run(c, steps[m])
            assert np.array_equal(b.get_state(m), ref["U"]) and infos[m].t == ref["t"]
