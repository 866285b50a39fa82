"""The spread 1D stage kernel (stage1d.cuh) runs with overlapped launches: a stage's blocks
are resident while the previous stage still writes the primitives they will read.

Stepped without a graph, an all-1D batch is one unbroken chain of such launches over several
steps; stepped as a graph, every step is a launch of its own.  Both must give the same bits.
A launch that overlaps its predecessor must not read primitives through the non-coherent
read-only path, which wants them unmodified while the kernel is resident: that is checked in
the source, where a CPU can see it.
"""
import os
import re

import numpy as np
import pytest

from grhd_b200 import build
from grhd_b200.problem import Problem
from grhd_b200.solver import GpuBatch, GpuGrid
from tests.helpers import initial_state, michel, shock_tube

GPU_SRC = os.path.join(build.CSRC, "gpu")


def test_overlapped_kernels_read_primitives_coherently():
    seen = 0
    for name in sorted(os.listdir(GPU_SRC)):
        text = open(os.path.join(GPU_SRC, name)).read()
        if "griddepcontrol.launch_dependents" not in text:
            continue
        seen += 1
        code = re.sub(r"//[^\n]*", "", text)
        assert not re.search(r"GRHD_LDP|__ldg\(\s*&?\s*(Pin|Pout)|\bld_prim\(|\bld_cell\b", code), name
        fills = re.findall(r"load_cell<([^>]*)>", code)
        assert fills and all(re.fullmatch(r"\s*\w+\s*,\s*true\s*", a) for a in fills), (name, fills)
    assert seen == 1


def _run(pbs, precision, graph, steps):
    import torch
    s = torch.cuda.Stream(device=0)
    grids = []
    for pb in pbs:
        g = GpuGrid(pb, precision=precision, upload_initial=False, stream=s.cuda_stream)
        g.upload(p=initial_state(pb))
        g.prim_to_cons()
        grids.append(g)
    out = []
    with GpuBatch(grids) as b:
        for k in range(len(grids)):
            b.set_clock(k, 0.0, 1e30, steps)
        b.step(steps, graph=graph)
        for k, g in enumerate(grids):
            out.append((*g.download(), g.counters(), b.clock(k)))
    for g in grids:
        g.close()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed_comp64", "mixed_comp32"])
def test_eager_chain_equals_graph_replays(precision):
    """Every boundary fill that reads an interior cell (outflow, periodic, dust, Michel's
    copy), one and several tiles, more steps than the rotation has buffers."""
    pbs = [shock_tube(nx=5), shock_tube(nx=200, rec="weno3", sensor=True), michel(nx=130),
           Problem.from_keys("convergence", nx=64), Problem.from_keys("dust", nx=127, nz=1)]
    eager, replay = _run(pbs, precision, False, 40), _run(pbs, precision, True, 40)
    for (up, p, cnt, clk), (up_g, p_g, cnt_g, clk_g) in zip(eager, replay):
        assert np.array_equal(up, up_g) and np.array_equal(p, p_g)
        assert cnt == cnt_g and clk == clk_g and clk[1] == 40
