"""The stage kernel's spread form for small launches of 1D grids (stage1d.cuh) against the
stage kernel's 256-cell tiles, bit for bit in FP64 (state, primitives, counters).

A small batch of 1D grids steps with the spread form; the same grids beside enough others to
pass its tile limit step with the 256-cell tiles.  Sizes sit around its tile of 63 cells and
its 64 faces, and below the stencil's reach; schemes, solvers, the shock sensor and boundary
cases cover its branches.  (The mixed policies' runs of 1D grids are held to their bars in
test_gpu_parity.py and test_gpu_batch.py, which step such grids with both forms.)
"""
import numpy as np
import pytest

from grhd_b200.problem import Problem
from grhd_b200.solver import GpuBatch, GpuGrid
from tests.helpers import initial_state, michel, shock_tube

pytestmark = pytest.mark.gpu

FILL = dict(nx=4096)  # 66 tiles of 63 cells each: five pass the limit of 296
STEPS = 12
PROBLEMS = {
    "weno5-hlle": lambda nx: shock_tube(nx=nx),
    "mp5-hllc-sensor": lambda nx: shock_tube(nx=nx, rec="mp5", rs="hllc", sensor=True),
    "weno5-hllc": lambda nx: shock_tube(nx=nx, rec="weno5", rs="hllc", sod_velocity_left=0.6, sod_velocity_right=-0.4),
    "weno3-hlle-sensor": lambda nx: shock_tube(nx=nx, rec="weno3", sensor=True),
    "tvd-hllc-sensor": lambda nx: shock_tube(nx=nx, rec="tvd", rs="hllc", sensor=True, tvd_limiter="superbee"),
    "godunov-hlle": lambda nx: shock_tube(nx=nx, rec="godunov"),
    "michel": lambda nx: michel(nx=nx),
    "dust-weno5-hllc": lambda nx: Problem.from_keys("dust", nx=nx, nz=1, reconstruction="weno5", riemann_solver="hllc"),
    "convergence": lambda nx: Problem.from_keys("convergence", nx=nx),
}


def _run(pbs, extra):
    import torch
    s = torch.cuda.Stream(device=0)
    grids = []
    for pb in pbs + extra:
        g = GpuGrid(pb, upload_initial=False, stream=s.cuda_stream)
        g.upload(p=initial_state(pb))
        g.prim_to_cons()
        grids.append(g)
    out = []
    with GpuBatch(grids) as b:
        for k in range(len(grids)):
            b.set_clock(k, 0.0, 1e30, STEPS)
        b.step(STEPS)
        for g in grids[:len(pbs)]:
            up, p = g.download()
            out.append((up, p, g.counters()))
    for g in grids:
        g.close()
    return out


@pytest.mark.parametrize("name", list(PROBLEMS))
def test_spread_form_matches_tiles(name):
    make = PROBLEMS[name]
    pbs = [make(nx) for nx in (5, 62, 63, 64, 66, 127, 200)]
    small = _run(pbs, [])
    large = _run(pbs, [make(FILL["nx"]) for _ in range(5)])
    for (up, p, cnt), (up_t, p_t, cnt_t) in zip(small, large):
        assert np.array_equal(up, up_t) and np.array_equal(p, p_t)
        assert cnt == cnt_t
