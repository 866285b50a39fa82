"""A 1D grid's result must not depend on which form of the stage kernel its batch picks: the
spread form (stage1d.cuh) while the batch's 1D tiles fit the GPU at once, the 256-cell tiles
beyond.  Every precision policy, bit for bit; each batch is checked to run the form meant (only
an all-spread step has no launch for its clocks).
"""
import zlib

import numpy as np
import pytest

from grhd_b200.problem import Problem
from grhd_b200.serve import GpuEngine, SolveServer, make_stream
from grhd_b200.solver import GpuBatch, GpuGrid
from tests.helpers import initial_state, michel, shock_tube

pytestmark = pytest.mark.gpu

PRECISIONS = ["fp64", "mixed", "mixed_comp64", "mixed_comp32"]
FILL = 4096  # 66 tiles of 63 cells: five pass the limit of 296
PROBLEMS = {}
for _rec in ("weno5", "mp5", "weno3", "tvd", "godunov"):
    PROBLEMS[f"tube-{_rec}"] = lambda nx, r=_rec: shock_tube(nx=nx, rec=r, sod_velocity_left=0.3)
    PROBLEMS[f"tube-{_rec}-sensor"] = lambda nx, r=_rec: shock_tube(nx=nx, rec=r, sensor=True)
    PROBLEMS[f"michel-{_rec}"] = lambda nx, r=_rec: michel(nx=nx, rec=r)
PROBLEMS["dust"] = lambda nx: Problem.from_keys("dust", nx=nx, nz=1, reconstruction="weno5")
PROBLEMS["convergence"] = lambda nx: Problem.from_keys("convergence", nx=nx)


def _wild(pb, seed):
    """Random primitives: densities and pressures over ten decades, down to below the floors,
    velocities up to 0.99 in any direction of the grid's coordinates."""
    rng = np.random.default_rng(seed)
    p = initial_state(pb).copy()
    n = p.shape[:-1]
    p[..., 0] = 10.0 ** rng.uniform(-9, 1, n)
    p[..., 1] = 10.0 ** rng.uniform(-11, 1, n)
    v = rng.normal(size=n + (3,))
    p[..., 2:] = v / np.linalg.norm(v, axis=-1, keepdims=True) * rng.uniform(0, 0.99, n)[..., None]
    return p


def _run(states, precision, steps, spread):
    import torch
    s = torch.cuda.Stream(device=0)
    fill = [] if spread else [(pb, initial_state(pb)) for pb in [shock_tube(nx=FILL)] * 5]
    grids, out = [], []
    for pb, p in states + fill:
        g = GpuGrid(pb, precision=precision, upload_initial=False, stream=s.cuda_stream)
        g.upload(p=p)
        g.prim_to_cons()
        grids.append(g)
    with GpuBatch(grids) as b:
        for k in range(len(grids)):
            b.set_clock(k, 0.0, 1e30, steps)
        b.step(steps)
        for g in grids[:len(states)]:
            out.append((*g.download(), g.counters()))
        assert ("advance_clocks" not in [n for n, _ in b.profile_step()]) == spread
    for g in grids:
        g.close()
    return out


@pytest.mark.parametrize("wild", [False, True], ids=["ordinary", "wild"])
@pytest.mark.parametrize("precision", PRECISIONS)
def test_forms_agree(precision, wild):
    for name, make in PROBLEMS.items():
        pbs = [make(nx) for nx in (5, 63, 64, 200)]
        seed = zlib.crc32(name.encode())
        states = [(pb, _wild(pb, seed + k) if wild else initial_state(pb)) for k, pb in enumerate(pbs)]
        steps = 3 if wild else 20
        for (up, p, cnt), (up_t, p_t, cnt_t) in zip(_run(states, precision, steps, True), _run(states, precision, steps, False)):
            assert np.array_equal(up, up_t, equal_nan=True), name
            assert np.array_equal(p, p_t, equal_nan=True), name
            assert cnt == cnt_t, name


@pytest.mark.parametrize("precision", ["mixed", "mixed_comp64", "mixed_comp32"])
def test_forms_agree_on_noisy_accretion(precision):
    """States that jump at every face, long enough for a difference of one rounding anywhere on
    the path to spread through the flow; the sonic point included."""
    states = []
    for k, rec in enumerate(("weno5", "mp5", "weno3", "tvd", "godunov")):
        pb = michel(nx=1000, rec=rec, perturbation_amplitude=0.05, perturbation_seed=100 + k)
        states.append((pb, initial_state(pb)))
    for (up, p, cnt), (up_t, p_t, cnt_t) in zip(_run(states, precision, 100, True), _run(states, precision, 100, False)):
        assert np.array_equal(up, up_t) and np.array_equal(p, p_t) and cnt == cnt_t


@pytest.mark.parametrize("precision", PRECISIONS)
def test_served_results_past_the_limit_equal_solo_runs(precision):
    reqs = make_stream(16, seed=5, rate=1e6, michel_final_time=0.25, riemann_final_time=0.01,
                       riemann_cells=(1000, 3000), michel_cells=(1000, 3000))
    tiles = [-(-r.cells // 63) for r in reqs]
    assert sum(tiles) > 296 and max(tiles) <= 296 and {r.kind for r in reqs} == {"riemann", "michel"}
    eng = GpuEngine(precision)
    srv = SolveServer(eng, steps_per_round=8, keep_results=True)
    res = srv.run(reqs)
    eng.close()
    assert srv.peak_active == len(reqs)
    for r, q in zip(res, reqs):
        pb = Problem.from_keys(q.problem, **q.keys)
        g = GpuGrid(pb, precision=precision, upload_initial=False)
        g.upload(p=pb.initial_prims())
        g.prim_to_cons()
        n, t = g.run(0.0, q.final_time)
        up = g.download(want_p=False)[0]
        g.close()
        assert (r.steps, r.t) == (n, t) and np.array_equal(r.up, up), f"request {q.id} ({q.kind}, {q.cells} cells)"
