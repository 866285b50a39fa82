"""State copies to and from host arrays that do not start at a multiple of 8 bytes: the copy
engines take any address, the layout kernels must not be handed such a one.  Page-locked and
pageable, below and above the size the kernels address directly."""
import ctypes as C

import numpy as np
import pytest

from grhd_b200.solver import GpuGrid
from tests.helpers import shock_tube

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pin", [True, False], ids=["page-locked", "pageable"])
@pytest.mark.parametrize("nx", [5, 257, 4000])
@pytest.mark.parametrize("offset", [4, 1])
def test_unaligned_state_copies(nx, offset, pin):
    import torch
    g = GpuGrid(shock_tube(nx=nx))
    n = 40 * nx
    want = np.random.default_rng(nx).uniform(1.0, 2.0, 5 * nx)
    buf = torch.zeros(n + 16, dtype=torch.uint8)
    buf = buf.pin_memory() if pin else buf
    raw = buf.numpy()
    at = (-buf.data_ptr()) % 8 + offset
    ptr = C.cast(buf.data_ptr() + at, C.POINTER(C.c_double))
    raw[at:at + n] = want.view(np.uint8)
    assert g.lib.grhd2_gpu_upload_async(g._h, ptr, None) == 0
    g.synchronize()
    assert np.array_equal(g.download(want_p=False)[0].ravel(), want)
    raw[...] = 0
    assert g.lib.grhd2_gpu_download_async(g._h, ptr, None) == 0
    g.synchronize()
    assert np.array_equal(raw[at:at + n], want.view(np.uint8))
    assert not raw[:at].any() and not raw[at + n:].any()
    g.close()
