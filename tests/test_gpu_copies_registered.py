"""State copies with host memory the caller registered itself: read and write, and read-only (an
upload's source; a download is the caller's error there and is not tried)."""
import ctypes as C
import mmap

import numpy as np
import pytest

from grhd_b200.solver import GpuGrid
from tests.helpers import shock_tube

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [200, 4000])
@pytest.mark.parametrize("readonly", [False, True])
def test_registered_state_copies(nx, readonly):
    import torch
    g = GpuGrid(shock_tube(nx=nx))
    size = -(-40 * nx // mmap.PAGESIZE) * mmap.PAGESIZE
    mem = mmap.mmap(-1, size)
    host = np.frombuffer(mem, dtype=np.float64)
    want = np.random.default_rng(nx).uniform(1.0, 2.0, 5 * nx)
    host[:5 * nx] = want
    cudart = torch.cuda.cudart()
    flags = 8 if readonly else 0  # cudaHostRegisterReadOnly
    assert int(cudart.cudaHostRegister(host.ctypes.data, size, flags)) == 0
    ptr = C.cast(host.ctypes.data, C.POINTER(C.c_double))
    assert g.lib.grhd2_gpu_upload_async(g._h, ptr, None) == 0
    g.synchronize()
    assert np.array_equal(g.download(want_p=False)[0].ravel(), want)
    if not readonly:
        host[:] = 0.0
        assert g.lib.grhd2_gpu_download_async(g._h, ptr, None) == 0
        g.synchronize()
        assert np.array_equal(host[:5 * nx], want) and not host[5 * nx:].any()
    assert int(cudart.cudaHostUnregister(host.ctypes.data)) == 0
    g.close()
