"""A launch that the runtime refuses (into a capture that something else has
invalidated) is answered with a status, and the calls after it succeed."""
import ctypes

import numpy as np
import pytest
import torch

import oracle_lib as O
from test_gpu_field import _lib  # noqa: F401
from provekit_b200._lib import PKG_ERR_CUDA, PKG_OK, lib

pytestmark = pytest.mark.gpu


def test_refused_launch_leaves_nothing_behind():
    L = lib()
    a = O.sample_fr(3, 1 << 10)
    d = torch.from_numpy(a.view(np.int64).copy()).cuda()
    leaves = torch.from_numpy(O.sample_fr(4, 3 << 7).view(np.uint8).reshape(-1).copy()).cuda()
    out = torch.zeros(32 * 255, dtype=torch.uint8, device="cuda")
    calls = {
        "transform": lambda s: L.pkg_ntt_nr(d.data_ptr(), 1 << 10, 1 << 10, 1, s),
        "fold": lambda s: L.pkg_skyscraper_hash_many(96, leaves.data_ptr(), 128, out.data_ptr(), s),
        "tree": lambda s: L.pkg_merkle_levels(out.data_ptr(), 128, s),
    }
    other = torch.cuda.Stream()
    for name, call in calls.items():
        assert call(other.cuda_stream) == PKG_OK, name
        torch.cuda.synchronize()
        s = torch.cuda.Stream()
        cuda = ctypes.CDLL("libcuda.so.1")
        stream = ctypes.c_void_p(s.cuda_stream)
        assert cuda.cuStreamBeginCapture_v2(stream, 2) == 0  # relaxed: for this stream only
        # a synchronisation is not allowed there and invalidates the capture
        assert cuda.cuStreamSynchronize(stream) != 0
        assert call(s.cuda_stream) == PKG_ERR_CUDA, name
        graph = ctypes.c_void_p()
        assert cuda.cuStreamEndCapture(stream, ctypes.byref(graph)) != 0
        assert call(other.cuda_stream) == PKG_OK, name
        torch.cuda.synchronize()
