"""The sizes by which GPU tests mean to reach one form of a kernel or the other do so: the limits
are read from the dispatch rules, so that a test does not pass by comparing a form with itself
when a limit moves."""
import inspect
import os
import re

from grhd_b200 import build
from tests import test_gpu_cell_blocks, test_gpu_stage1d, test_gpu_stage1d_forms

SRC = open(os.path.join(build.CSRC, "gpu", "grhd2_gpu.cu")).read()
LAUNCH = open(os.path.join(build.CSRC, "gpu", "flux_launch.h")).read()


def _const(text, name):
    return eval(re.search(rf"constexpr int {name} = ([0-9 *]+);", text).group(1))


def test_spread_1d_limit():
    limit, cells = _const(SRC, "STAGE1D_TILES_MAX"), _const(LAUNCH, "STAGE1D_CELLS")
    small = sum(-(-nx // cells) for nx in (5, 62, 63, 64, 66, 127, 200))
    assert small <= limit < 5 * -(-test_gpu_stage1d.FILL["nx"] // cells)
    assert limit < 5 * -(-test_gpu_stage1d_forms.FILL // cells)
    assert "(5, 62, 63, 64, 66, 127, 200)" in inspect.getsource(test_gpu_stage1d)


def test_wide_cell_limit():
    limit = _const(SRC, "WIDE_CELLS_FROM_BLOCKS")
    assert "20LL * CELL_BS_WIDE * grp.nb[K_CELL_WIDE] > 21LL * CELL_BS * grp.nb[K_CELL]" in SRC

    def blocks(kw, rows):  # 32 cells along i, `rows` along k
        return -(-kw["nx"] // 32) * kw.get("ny", 1) * -(-kw["nz"] // rows)

    mark = next(m for m in test_gpu_cell_blocks.test_wide_blocks_match_narrow.pytestmark if m.name == "parametrize")
    for _, sizes in mark.args[1]:
        wide, narrow = (sum(blocks(kw, rows) for kw in sizes) for rows in (8, 4))
        assert wide >= limit and 20 * 256 * wide <= 21 * 128 * narrow  # the batch takes the wide form
        assert all(blocks(kw, 8) < limit for kw in sizes[:-1])  # each grid compared alone, but the largest, does not
        assert sum(kw["nx"] * kw.get("ny", 1) * kw["nz"] for kw in sizes) < 2_000_000  # one scheme group, not two
