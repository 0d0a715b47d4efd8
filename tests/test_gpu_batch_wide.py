"""Batches beyond the lines between two forms, against the plain entry points: a
job of 2^17 among small ones (a tree level of more than 2^15 nodes in tiles,
sumcheck rounds of more than 2^14 pairs with a thread per pair for all jobs),
and counts of jobs that leave the last CTA of the transcripts partly empty."""
import pytest
import torch

from test_gpu_batch import _lib, check_batch  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[5, 17, 9, 4, 12], [17], [10, 4, 6], [16, 16, 15, 7, 11, 16, 4]])
@pytest.mark.parametrize("use_graph", [False, True])
def test_matches_plain(sizes, use_graph):
    from provekit_b200.batch import Batch
    b = Batch(sizes, seed=31 + len(sizes))
    s = torch.cuda.Stream()
    b.run(use_graph=use_graph, stream=s)
    b.run(use_graph=use_graph, stream=s)
    s.synchronize()
    check_batch(b)
    b.close()
