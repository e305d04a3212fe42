"""Edges between two water films of which one is exactly as deep as the threshold below which a first-order
scheme takes a depth for dry: the reference's two evaluations of such an edge are not mirror images of one
another, and each side's flux is the one of its own."""
import numpy as np
import pytest

import harness as H
from cuteflow_gb300 import cases

EPS = {1: float(np.float32(1e-8)), 2: float(np.float32(1e-6))}


def _films(nx, ny, iflux, seed):
    c = cases.lake_at_rest(nx, ny, seed=seed, iflux=iflux)
    c.z = np.zeros(c.z.size)
    rng = np.random.default_rng(seed)
    e = EPS[iflux]
    h = rng.choice([0.0, e, 0.5 * e, np.nextafter(e, 0), np.nextafter(e, 1), 0.3], c.nelt)
    c.U0 = np.stack([h, h * rng.choice([0.0, 1.0, -0.7], c.nelt), h * rng.choice([0.0, 0.4, -1.0], c.nelt)], 1)
    c.params["tolisec"] = 0.1 * e
    return c


@pytest.mark.parametrize("xd", [0, 1, 2])
@pytest.mark.parametrize("iflux", [1, 2])
def test_films_are_the_oracles(oracle, iflux, xd):
    for seed in (1, 2):
        c = _films(23, 11, iflux, seed)
        H.set_xd(xd)
        try:
            f, _ = H.edge_fluxes(c, c.U0, 0.01)
        finally:
            H.set_xd(0)
        assert np.array_equal(f, oracle.edge_fluxes(c, c.U0, 0.01))


@pytest.mark.gpu
@pytest.mark.parametrize("iflux", [1, 2])
def test_films_on_the_gpu(gpu_lib, oracle, iflux):
    from cuteflow_gb300 import Solver
    c = _films(17, 9, iflux, 3)
    ref = oracle.run(c, 2, check=False)
    for tuning in ((0, 0), (1, 0), (1, 0x1F)):
        with Solver(c) as s:
            s.set_tuning(*tuning)
            s.set_state(c.U0)
            info = s.step(2, check=False)
            assert np.array_equal(s.get_state(), ref["U"]) and info.t == ref["t"]
