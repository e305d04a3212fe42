"""A part's step under every arithmetic setting, the partial ones included, against the undivided run."""
import multiprocessing as mp
import os
import sys

import numpy as np
import pytest

from cuteflow_gb300 import domains
from test_gpu_domains import ROOT, _case, _free_port

pytestmark = pytest.mark.gpu

TUNINGS = [(0, 0), (1, 0), (1, 0x2), (1, 0x5), (1, 0x15), (1, 0x17), (1, 0x1F)]


def _rank(rank, world, kind, nsteps, port, out):
    sys.path[:0] = [ROOT, os.path.dirname(os.path.abspath(__file__))]
    import torch
    import torch.distributed as dist
    torch.cuda.set_device(0)
    dist.init_process_group("gloo", init_method=f"tcp://127.0.0.1:{port}", rank=rank, world_size=world)
    try:
        c, prm = _case(kind)
        r = domains.PartRunner(c, world, rank, dist, params=prm)
        for tuning in TUNINGS:
            r.solver.set_tuning(*tuning)
            r.set_state(np.asarray(c.U0, dtype=np.float64))
            info = r.step(nsteps)
            out.put((rank, tuning, r.get_owned_state(), info.t))
        r.close()
    finally:
        dist.destroy_process_group()


@pytest.mark.parametrize("kind", ["flood_hllc", "flood_waf", "channel_muscl"])
def test_partial_masks_on_parts(gpu_lib, kind):
    from cuteflow_gb300 import Solver
    world, nsteps = 2, 12
    c, prm = _case(kind)
    with Solver(c, prm) as s:
        s.set_state(c.U0)
        t_ref = s.step(nsteps).t
        ref = s.get_state()
    ctx = mp.get_context("spawn")
    out = ctx.Queue()
    port = _free_port()
    procs = [ctx.Process(target=_rank, args=(r, world, kind, nsteps, port, out), daemon=True) for r in range(world)]
    for pr in procs:
        pr.start()
    got = [out.get(timeout=300) for _ in range(world * len(TUNINGS))]
    for pr in procs:
        pr.join(timeout=60)
        assert pr.exitcode == 0
    parts = domains.partition(c, world, prm)
    for rank, tuning, U, t in got:
        assert t == t_ref and np.array_equal(U, ref[parts[rank].owned]), (rank, tuning)
