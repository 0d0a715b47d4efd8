"""GPU parity of WHIR sumcheck rounds on both sides of the size where four lanes
take a pair (2^14 pairs), and at one pair, with and without folding, word for
word against the oracle; the tables hold the ends of the range (0, p - 1) among
random values.  (Spartan rounds: whole sumchecks up to 2^20 entries in
test_gpu_spartan.py pass through every size.)"""
import numpy as np
import pytest
import torch

import oracle_lib as O
from fieldutil import P, to_limbs
from test_gpu_field import _lib  # noqa: F401
from provekit_b200.whir import sumcheck_round

pytestmark = pytest.mark.gpu


def table(n, seed):
    v = O.sample_fr(seed, n)
    v[: n // 4] = np.array(to_limbs(P - 1), np.uint64)
    v[n // 2: n // 2 + n // 8] = 0
    return v


@pytest.mark.parametrize("fold", [False, True])
@pytest.mark.parametrize("log_pairs", [0, 5, 6, 7, 14, 15])
def test_whir_round(log_pairs, fold):
    size = (4 if fold else 2) << log_pairs
    f, w = table(size, 1 + log_pairs), table(size, 50 + log_pairs)
    alpha = O.sample_fr(9, 1)[0] if fold else None
    df, dw = (torch.from_numpy(x.view(np.int64).copy()).cuda() for x in (f, w))
    got = sumcheck_round(df, dw, size, alpha)
    exp = O.whir_sumcheck_round(f, w, size, alpha)
    assert np.array_equal(got, exp)
    live = size // 2 if fold else size  # folded in place by both
    assert np.array_equal(df.cpu().numpy().view(np.uint64)[:live], f[:live])
    assert np.array_equal(dw.cpu().numpy().view(np.uint64)[:live], w[:live])
