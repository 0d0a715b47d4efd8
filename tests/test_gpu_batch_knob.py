"""The deprecated butterflies-per-thread value is kept and reported, and does not
cost a batch its plan: the captured graph is replayed after it is set (on the
default stream, where a graph can be launched but not captured)."""
import pytest
import torch

from test_gpu_batch import _lib, check_batch  # noqa: F401

pytestmark = pytest.mark.gpu


def test_graph_stays():
    from provekit_b200._lib import check, lib
    from provekit_b200.batch import Batch
    b = Batch([6, 9, 4], seed=8)
    s = torch.cuda.Stream()
    b.run(use_graph=True, stream=s)
    s.synchronize()
    k, e, _ = b.params()
    for lb in (0, 1, 2):
        check(lib().pkg_batch_set_butterflies_per_thread(b._b, lb))
        assert b.params() == (k, e, lb)
        b.run(use_graph=True, stream=torch.cuda.default_stream())
        torch.cuda.synchronize()
    check_batch(b)
    b.close()
