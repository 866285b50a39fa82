"""The mixed policies' result must not depend on the face-kernel variant, which a batch picks by
its size: 'split', 'split_var' and 'fused' agree to the bit on x-z, x-y and 3D grids, for every
scheme and both Riemann solvers, on ordinary and on random states."""
import zlib

import numpy as np
import pytest

from grhd_b200.problem import Problem
from grhd_b200.solver import GpuBatch, GpuGrid
from tests.helpers import initial_state, torus_2p5d, torus_3d
from tests.test_gpu_stage1d_forms import _wild

pytestmark = pytest.mark.gpu

SHAPES = {
    "xz": lambda rec, rs, s: torus_2p5d(nx=37, nz=19, rec=rec, rs=rs, sensor=s),
    "xy": lambda rec, rs, s: Problem.from_keys("fishbone_sagittal", nx=37, ny=21, reconstruction=rec, riemann_solver=rs,
                                               shock_sensor=s, perturbation="pressure_noise",
                                               perturbation_amplitude=0.05, perturbation_time=0.0, perturbation_seed=9),
    "3d": lambda rec, rs, s: torus_3d(nx=20, ny=8, nz=10, rec=rec, rs=rs, sensor=s),
    "kh": lambda rec, rs, s: Problem.from_keys("kelvin_helmholtz", nx=33, nz=40, reconstruction=rec, riemann_solver=rs,
                                               shock_sensor=s, perturbation="pressure_noise",
                                               perturbation_amplitude=0.05, perturbation_time=0.0, perturbation_seed=9),
}


def _run(pb, p, variant, steps):
    import torch
    s = torch.cuda.Stream(device=0)
    g = GpuGrid(pb, precision="mixed", upload_initial=False, stream=s.cuda_stream)
    g.upload(p=p)
    g.prim_to_cons()
    with GpuBatch([g]) as b:
        b.set_flux_variant(variant)
        b.set_clock(0, 0.0, 1e30, steps)
        b.step(steps)
        out = (*g.download(), g.counters())
    g.close()
    return out


@pytest.mark.parametrize("shape", list(SHAPES))
@pytest.mark.parametrize("rs", ["hlle", "hllc"])
@pytest.mark.parametrize("rec", ["weno5", "mp5", "weno3", "tvd", "godunov"])
def test_variants_agree(shape, rs, rec):
    for sensor in (False, True):
        pb = SHAPES[shape](rec, rs, sensor)
        for wild, steps in ((False, 12), (True, 2)):
            p = _wild(pb, zlib.crc32(f"{shape}{rs}{rec}{sensor}".encode())) if wild else initial_state(pb)
            up, pr, cnt = _run(pb, p, "split", steps)
            for variant in ("split_var", "fused"):
                u, q, c = _run(pb, p, variant, steps)
                assert np.array_equal(u, up, equal_nan=True) and np.array_equal(q, pr, equal_nan=True), (variant, sensor, wild)
                assert c == cnt, (variant, sensor, wild)
