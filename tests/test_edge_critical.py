"""WAF where a wave stands still: critical and colliding flows whose wave speeds are exactly 0, on a mesh of
axis-parallel edges.  WAF's weights take the sign of the speed, and that of a zero is the one that the
reference's evaluation from the side's own element gives."""
import numpy as np
import pytest

import harness as H
from cuteflow_gb300 import cases


def _critical(iflux, seed, limiter):
    c = cases.lake_at_rest(23, 11, seed=1, iflux=iflux)
    c.x, c.y = cases.grid_mesh(23, 11, 23.0, 11.0, 1, 0.0)[:2]
    c.z = np.zeros(c.z.size)
    rng = np.random.default_rng(seed)
    g = (9.81, 1.0, 4.0)[seed % 3]
    h = np.full(c.nelt, (1.0, 0.25)[seed % 2])
    s = np.sqrt(g * h)
    c.U0 = np.stack([h, h * s * rng.choice([1.0, -1.0, 2.0, 0.0], c.nelt), h * s * rng.choice([1.0, 0.0, -1.0], c.nelt)], 1)
    c.U0[rng.random(c.nelt) < 0.2] = 0.0
    c.params.update(gp=g, ilimiteur=limiter)
    return c


@pytest.mark.parametrize("xd", [0, 1, 2])
@pytest.mark.parametrize("limiter", [0, 1, 2, 3, 4])
def test_standing_waves_are_the_oracles(oracle, limiter, xd):
    for seed in range(6):
        c = _critical(3, seed, limiter)
        H.set_xd(xd)
        try:
            f, _ = H.edge_fluxes(c, c.U0, 0.05)
        finally:
            H.set_xd(0)
        assert np.array_equal(f, oracle.edge_fluxes(c, c.U0, 0.05))


@pytest.mark.gpu
@pytest.mark.parametrize("iflux", [1, 2, 3, 4])
def test_standing_waves_on_the_gpu(gpu_lib, oracle, iflux):
    from cuteflow_gb300 import Solver
    c = _critical(iflux, 1, 1)
    ref = oracle.run(c, 3, check=False)
    for tuning in ((0, 0), (1, 0), (1, 0x1F)):
        with Solver(c) as s:
            s.set_tuning(*tuning)
            s.set_state(c.U0)
            info = s.step(3, check=False)
            assert np.array_equal(s.get_state(), ref["U"]) and info.t == ref["t"]
