"""The two-sided edge evaluation where it can go wrong: nearly dry elements (depths at and around the
dry threshold, whose raw and masked reconstructions differ), beds of equal and very unequal height, and
meshes of a few edges (partial warps and tiles)."""
import numpy as np
import pytest

import harness as H
from cuteflow_gb300 import cases


def _shallow(nx, ny, iflux, seed, tolisec=1e-3):
    """A walled basin whose depths lie at, just around and far from tolisec."""
    c = cases.lake_at_rest(nx, ny, seed=seed, iflux=iflux)
    rng = np.random.default_rng(seed)
    c.z = np.where(rng.random(c.z.size) < 0.5, 0.0, c.z)
    pick = rng.integers(0, 6, c.nelt)
    h = np.select([pick == 0, pick == 1, pick == 2, pick == 3], [0.0, tolisec, tolisec * (1 + 1e-15), 0.6 * tolisec],
                  rng.uniform(0.002, 0.6, c.nelt))
    c.U0 = np.stack([h, h * rng.normal(size=c.nelt), h * rng.normal(size=c.nelt)], 1)
    c.params["tolisec"] = tolisec
    return c


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("iflux", [1, 2, 3, 4])
def test_nearly_dry_edges_are_the_oracles(oracle, iflux, mode):
    c = _shallow(23, 11, iflux, 5)
    H.set_xd(mode)
    try:
        f, _ = H.edge_fluxes(c, c.U0, 0.01)
    finally:
        H.set_xd(0)
    assert np.array_equal(f, oracle.edge_fluxes(c, c.U0, 0.01))


@pytest.mark.gpu
@pytest.mark.parametrize("iflux", [1, 2, 3, 4])
@pytest.mark.parametrize("size", [(1, 1), (3, 2), (7, 6), (43, 1), (23, 11)])
def test_small_meshes_on_the_gpu(gpu_lib, oracle, iflux, size):
    from cuteflow_gb300 import Solver
    for flux_mode in (0, 1):
        c = _shallow(*size, iflux, 7)
        c.params["flux_mode"] = flux_mode
        ref = oracle.run(c, 6, check=False)
        for tuning in ((0, 0), (1, 0), (1, 0x1F)):
            with Solver(c) as s:
                s.set_tuning(*tuning)
                s.set_state(c.U0)
                info = s.step(6, check=False)
                assert np.array_equal(s.get_state(), ref["U"]) and info.t == ref["t"], (tuning, flux_mode)
