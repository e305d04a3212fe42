"""Inlet sums and discharge sums between the steps of a graph: lists shorter than a warp, longer than a
warp and longer than a block, and members that need only one of the two, or neither."""
import numpy as np
import pytest

from cuteflow_gb300 import cases

pytestmark = pytest.mark.gpu

STEADY = dict(tol_reg_perm=1e-9, steady_count=1000)


@pytest.mark.parametrize("ny", [4, 17, 33, 150, 300])
def test_sums_over_lists_of_any_length(gpu_lib, oracle, ny):
    from cuteflow_gb300 import Solver
    c = cases.channel(nx=10, ny=ny, ly=10.0 * ny, inlet=3)
    ref = oracle.run(c, 43, params=STEADY, check=False)
    with Solver(c, STEADY) as s:
        s.set_state(c.U0)
        for n in (1, 37, 5):
            info = s.step(n)
        U = s.get_state()
    assert np.array_equal(U, ref["U"]) and info.t == ref["t"]
    # sums of up to 300 terms of one sign, in another order: 300 units of the last place
    assert abs(info.q_in - ref["q_in"]) <= 300 * 2.3e-16 * abs(ref["q_in"])


def test_members_of_every_kind(gpu_lib):
    from cuteflow_gb300 import Batch, Solver
    cs = [cases.channel(nx=30, ny=n, inlet=i) for n, i in ((12, 3), (20, 2), (7, 3), (9, 2))]
    prm = [STEADY, STEADY, {}, {}]
    one = []
    for c, p in zip(cs, prm):
        with Solver(c, p) as s:
            s.set_state(c.U0)
            info = s.step(50)
            one.append((s.get_state(), info.t, info.q_in, info.q_out))
    with Batch(cs, prm) as b:
        for m, c in enumerate(cs):
            b.set_state(m, c.U0)
        infos = b.step(50)
        for m, (U, t, qi, qo) in enumerate(one):
            assert np.array_equal(b.get_state(m), U)
            assert (infos[m].t, infos[m].q_in, infos[m].q_out) == (t, qi, qo)
