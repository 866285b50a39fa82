"""The parts of a ghosted primitive array that an upload copies (prims_copy.h): every entry the
device layout kernel reads, inside the array, in copies the CUDA runtime takes -- the pitch of a
2D copy is limited to 2^31 - 1 bytes, which a plane of a large grid passes."""
import os
import subprocess

import numpy as np
import pytest

from grhd_b200 import build

MAIN = r"""
#include "prims_copy.h"
#include <cstdio>
#include <cstdlib>
int main(int, char **a) {
  return grhd::prims_in_pieces(atoi(a[1]), atoi(a[2]), atoi(a[3]), atoi(a[4]), [](const grhd::CopyPiece &x) {
    std::printf("%zu %zu %zu %zu\n", x.offset, x.pitch, x.width, x.rows);
    return 0;
  });
}
"""


@pytest.fixture(scope="module")
def pieces(tmp_path_factory):
    d = tmp_path_factory.mktemp("prims_copy")
    src, exe = d / "main.cpp", d / "main"
    src.write_text(MAIN)
    subprocess.run([build._cxx(), "-std=c++17", "-O1", "-I", os.path.join(build.CSRC, "gpu"), "-o", exe, src], check=True)

    def run(nx, ny, nz, ng):
        out = subprocess.run([exe, *map(str, (nx, ny, nz, ng))], check=True, capture_output=True, text=True).stdout
        return [tuple(map(int, line.split())) for line in out.splitlines()]
    return run


@pytest.mark.parametrize("shape", [(5, 1, 1), (7, 1, 4), (6, 5, 1), (4, 3, 6), (9, 2, 2)])
@pytest.mark.parametrize("ng", [1, 2, 3])
def test_pieces_cover_what_is_read(pieces, shape, ng):
    nx, ny, nz = shape
    dims = [n + 2 * ng + 1 for n in (nz, ny, nx)]
    got = np.zeros(int(np.prod(dims)) * 5 * 8, dtype=int)
    for off, pitch, width, rows in pieces(nx, ny, nz, ng):
        for r in range(rows):
            got[off + r * pitch:off + r * pitch + width] += 1
            assert off + r * pitch + width <= got.size
    got = got.reshape(*dims, 40)
    assert got.max() == 1
    k, j, i = np.ix_(*[np.arange(-ng, n + ng + 1) for n in (nz, ny, nx)])
    ins = [(x >= 1) & (x <= n) for x, n in ((i, nx), (j, ny), (k, nz))]
    read = ins[0] & ins[1] & ins[2]
    if ng == 2:  # the slabs at -nghost
        read = read | ((i == -ng) & ins[1] & ins[2]) | (ins[0] & (j == -ng) & ins[2] & (ny > 1)) \
            | (ins[0] & ins[1] & (k == -ng) & (nz > 1))
    assert got[np.broadcast_to(read, got.shape[:3])].all()


@pytest.mark.parametrize("shape", [(13_500_000, 1, 2), (7_500, 7_500, 4), (7_300, 7_300, 3), (54_000_000, 3, 2)])
@pytest.mark.parametrize("ng", [1, 2, 3])
def test_large_planes_stay_within_the_pitch(pieces, shape, ng):
    nx, ny, nz = shape
    row = 40 * (nx + 2 * ng + 1)
    plane = row * (ny + 2 * ng + 1)
    want = sum(row * n for n in [ny * nz] + ([nz] if ng == 2 and ny > 1 else []) + ([ny] if ng == 2 and nz > 1 else []))
    got = pieces(nx, ny, nz, ng)
    assert sum(w * r for _, _, w, r in got) == want
    for off, pitch, width, rows in got:
        assert rows == 1 or pitch <= 2**31 - 1
        assert off + (rows - 1) * pitch + width <= plane * (nz + 2 * ng + 1)
    firsts = {off for off, _, _, rows in got if rows == 1}
    if plane > 2**31 - 1:
        assert {row * (1 + ng) + plane * (k + ng) for k in range(1, nz + 1)} <= firsts
