"""Large states read into pageable and pinned host memory: the threaded copy
(above 32 MB, pageable) returns the same bytes as the runtime's."""
import ctypes

import numpy as np
import pytest
import torch

from viral_b200 import _abi as A
from viral_b200 import configs as C
from viral_b200.hydro import Hydro

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(66, 58, 50), (67, 61, 53), (130, 103, 21), (40, 30, 8)])
def test_same_bytes(nx, ny, nz):
    cfg = C.glauber_config(nx=nx, ny=ny, nz=nz)
    n = (nx + 6) * (ny + 6) * (nz + 6)
    want = np.random.default_rng(nx).standard_normal((18, n))
    with Hydro(cfg) as h:
        h.set_state(want, cfg.tau0)
        pinned = torch.empty(18, n, dtype=torch.float64).pin_memory()
        for _ in range(2):
            assert np.array_equal(h.get_state(), want)
            A.check(A.lib().vh_get_state(h.h, ctypes.cast(pinned.data_ptr(), A._dp)), h.h)
            assert np.array_equal(pinned.numpy(), want)
        odd = np.zeros(18 * n + 1)[1:]  # 8 bytes off the allocation's alignment
        A.check(A.lib().vh_get_state(h.h, odd.ctypes.data_as(A._dp)), h.h)
        assert np.array_equal(odd.reshape(18, n), want)
