"""The FP64 cell update in 256-thread blocks (used for scheme groups large enough to fill the
GPU) computes what the 128-thread blocks compute.

A batch is made large by a big grid; the small grids beside it have extents along k around
the wide tile's 8 rows and along i around its 32 columns.  Each must end in the state, the
primitives and the counters it has alone (128-thread blocks), bit for bit.
"""
import numpy as np
import pytest

from grhd_b200.solver import GpuBatch, GpuGrid
from tests.helpers import initial_state, torus_2p5d, torus_3d

pytestmark = pytest.mark.gpu


def _grid(pb, stream):
    g = GpuGrid(pb, upload_initial=False, stream=stream.cuda_stream)
    g.upload(p=initial_state(pb))
    g.prim_to_cons()
    return g


@pytest.mark.parametrize("make,sizes", [
    (torus_2p5d, [dict(nx=33, nz=7), dict(nx=31, nz=8), dict(nx=64, nz=9), dict(nx=40, nz=17), dict(nx=720, nz=240)]),
    (torus_3d, [dict(nx=33, ny=5, nz=6), dict(nx=32, ny=4, nz=8), dict(nx=20, ny=9, nz=10), dict(nx=96, ny=60, nz=64)]),
], ids=["xz", "3d"])
def test_wide_blocks_match_narrow(make, sizes):
    import torch
    s = torch.cuda.Stream(device=0)
    pbs = [make(**kw) for kw in sizes]
    alone = []
    for pb in pbs:
        g = _grid(pb, s)
        with GpuBatch([g]) as b:
            b.set_clock(0, 0.0, 1e30, 5)
            b.step(5)
            alone.append((*g.download(), g.counters()))
        g.close()
    grids = [_grid(pb, s) for pb in pbs]
    with GpuBatch(grids) as b:
        for k in range(len(grids)):
            b.set_clock(k, 0.0, 1e30, 5)
        b.step(5)
        for g, (up, p, cnt) in zip(grids, alone):
            up_b, p_b = g.download()
            assert np.array_equal(up_b, up) and np.array_equal(p_b, p)
            assert g.counters() == cnt
    for g in grids:
        g.close()
