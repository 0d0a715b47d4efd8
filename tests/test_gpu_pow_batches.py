"""The proof-of-work search beyond its first batch of 2^13 candidates (the later ones
run in tiles): nonces in the first, second and third batch, against the oracle, one
after the other on the words that a search leaves for the next."""
import numpy as np
import pytest

import oracle_lib as O
from test_gpu_field import _lib  # noqa: F401
from provekit_b200.skyscraper import pow_solve

pytestmark = pytest.mark.gpu

FIRST, SECOND = 1 << 13, 1 << 15  # candidates of a batch


def test_batches():
    seen = set()
    for top, challenge in ((1 << 47, [42, 43, 44, 45]), (1 << 47, [1, 2, 3, 4]),
                           (1 << 52, [42, 43, 44, 45]), (1 << 45, [5, 6, 7, 8]),
                           (1 << 47, [9, 9, 9, 9]), ((1 << 64) - 1, [9, 9, 9, 9])):
        threshold = [0, 0, 0, top]
        exp = O.lib().pko_sky_pow_solve(O.p64(np.array(challenge, np.uint64)),
                                        O.p64(np.array(threshold, np.uint64)))
        assert pow_solve(challenge, threshold) == exp
        seen.add((exp >= FIRST) + (exp >= FIRST + SECOND))
    assert seen == {0, 1, 2}
