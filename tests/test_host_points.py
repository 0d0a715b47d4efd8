"""The entry points that take points from the host answer a null or a device pointer
in their place with a status."""
import ctypes

import numpy as np
import pytest
import torch

from provekit_b200 import build
from provekit_b200._lib import PKG_ERR_INVALID_ARGUMENT, PKG_OK, lib


@pytest.fixture(scope="module")
def L():
    build.build()
    return lib()


def test_null_points(L):
    aligned = ctypes.c_void_p(1 << 20)  # checked, not read: the points are refused first
    assert L.pkg_eq_hypercube(None, 3, 8, aligned, None) == PKG_ERR_INVALID_ARGUMENT
    assert L.pkg_eq_accumulate(aligned, 3, None, aligned, 1, None) == PKG_ERR_INVALID_ARGUMENT


@pytest.mark.gpu
def test_device_points(L):
    host = np.zeros((3, 4), np.uint64)
    points = torch.zeros((3, 4), dtype=torch.int64, device="cuda")
    out = torch.zeros((8, 4), dtype=torch.int64, device="cuda")
    pinned = torch.zeros((3, 4), dtype=torch.int64).pin_memory()
    s = torch.cuda.current_stream().cuda_stream
    assert L.pkg_eq_hypercube(points.data_ptr(), 3, 8, out.data_ptr(), s) == PKG_ERR_INVALID_ARGUMENT
    for p, c in ((points.data_ptr(), host.ctypes.data), (host.ctypes.data, points.data_ptr())):
        assert L.pkg_eq_accumulate(out.data_ptr(), 3, p, c, 1, s) == PKG_ERR_INVALID_ARGUMENT
    for p in (host.ctypes.data, pinned.data_ptr()):
        assert L.pkg_eq_hypercube(p, 3, 8, out.data_ptr(), s) == PKG_OK
        assert L.pkg_eq_accumulate(out.data_ptr(), 3, p, p, 1, s) == PKG_OK
    assert L.pkg_eq_hypercube(None, 0, 1, out.data_ptr(), s) == PKG_OK
