"""Copies of the state between host and device by every route: pageable memory, page-locked
memory small enough for the layout kernels to address it themselves (128 KiB), and larger
page-locked memory, with arrays that do and do not start on a 16-byte boundary.  All must
move the same bytes.  The ghosted primitives'
upload, which skips the ghost planes, is held to the oracle by test_gpu_cases.py (the schemes
that read the -nghost slabs included); here the skipped planes may hold anything.
"""
import ctypes as C

import numpy as np
import pytest

from grhd_b200 import native as N
from grhd_b200.problem import Problem
from grhd_b200.solver import GpuGrid
from tests.helpers import initial_state, shock_tube, torus_2p5d, torus_3d

pytestmark = pytest.mark.gpu


def _ptr(t, offset):
    return C.cast(t.data_ptr() + 8 * offset, C.POINTER(C.c_double))


@pytest.mark.parametrize("nx", [5, 256, 257, 3276, 3277, 40000])  # 3276 cells: the last below 128 KiB
@pytest.mark.parametrize("offset", [0, 1])
def test_state_copies_agree(nx, offset):
    import torch
    pb = shock_tube(nx=nx)
    g = GpuGrid(pb)
    lib, n = g.lib, 5 * nx
    rng = np.random.default_rng(nx)
    want = rng.uniform(1.0, 2.0, n)
    pinned = torch.empty(n + 2, dtype=torch.float64).pin_memory()
    view = pinned.numpy()[offset:offset + n]
    view[...] = want
    assert lib.grhd2_gpu_upload_async(g._h, _ptr(pinned, offset), None) == 0
    assert np.array_equal(g.download(want_p=False)[0].ravel(), want)  # pageable download
    g.upload(up=want[::-1].copy())  # pageable upload
    pinned.numpy()[...] = 0.0
    assert lib.grhd2_gpu_download_async(g._h, _ptr(pinned, offset), None) == 0
    g.synchronize()
    assert np.array_equal(view, want[::-1])
    rest = np.delete(pinned.numpy(), np.arange(offset, offset + n))
    assert not rest.any()  # nothing beside the array
    g.close()


@pytest.mark.parametrize("make", [
    lambda: torus_2p5d(nx=33, nz=9), lambda: torus_3d(nx=20, ny=8, nz=6), lambda: shock_tube(nx=70),
    lambda: Problem.from_keys("fishbone_sagittal", nx=24, ny=11, reconstruction="weno3"),
    lambda: torus_3d(nx=16, ny=7, nz=6, rec="weno3", rs="hlle"),
    lambda: torus_2p5d(nx=24, nz=7, rec="tvd", sensor=True),
], ids=["xz", "3d", "1d", "xy-ng2", "3d-ng2", "xz-ng2"])
def test_primitive_upload_ignores_corner_ghosts(make):
    """Ghost cells outside the domain in two directions, and every ghost the boundary fill
    replaces, do not reach the device: NaN there changes nothing."""
    pb = make()
    p0 = initial_state(pb)
    g = GpuGrid(pb, upload_initial=False)
    g.upload(p=p0)
    ref = g.calc_rhs()
    ng = pb.ng
    bad = np.full_like(p0, np.nan)
    idx = [np.arange(-ng, n + ng + 1) for n in (pb.nz, pb.ny, pb.nx)]
    inside = [(i >= 1) & (i <= n) for i, n in zip(idx, (pb.nz, pb.ny, pb.nx))]
    keep = [a | (i == -ng) for a, i in zip(inside, idx)]  # the slabs at -nghost are read with two ghost cells
    mask = np.ix_(*[np.flatnonzero(k) for k in keep])
    bad[mask] = p0[mask]
    g.upload(p=np.zeros_like(p0) + 1.0)  # overwrite what the staging buffer held
    g.upload(p=bad)
    assert np.array_equal(g.calc_rhs(), ref)
    g.close()
