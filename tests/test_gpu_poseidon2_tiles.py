"""GPU parity of the tiled Poseidon2 permutation at the edges of its tiles (one
state, a tile less one, one more) and of its value range (0 and p - 1 in every
place), and of the sponge at every remainder of its rate, word for word
against the oracle."""
import numpy as np
import pytest
import torch

import oracle_lib as O
from fieldutil import P, to_limbs
from test_gpu_field import _lib  # noqa: F401
from provekit_b200.poseidon2 import poseidon2_hash_many, poseidon2_permutation_many

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int64).copy()).cuda()


def states(n, seed):
    v = O.sample_fr(seed, 4 * n)
    edge = np.array([to_limbs(x) for x in (0, P - 1, 1, P - 2)], np.uint64)
    v[:4] = edge[1]
    for i in range(1, min(n, 17)):
        v[4 * i:4 * i + 4] = edge[[(i >> (2 * k)) & 3 if k < 2 else i & 1 for k in range(4)]]
    return v


@pytest.mark.parametrize("n", [1, 127, 129, 1000])
def test_permutation(n):
    v = states(n, n)
    got = poseidon2_permutation_many(dev(v)).cpu().numpy().view(np.uint64)
    for i in range(n):
        e = np.ascontiguousarray(v[4 * i:4 * i + 4])
        O.lib().pko_poseidon2_permutation(O.p64(e))
        assert np.array_equal(got[4 * i:4 * i + 4], e), i


@pytest.mark.parametrize("length", [1, 2, 3, 4, 5, 6, 7])
def test_hash(length):
    n = 130
    v = states(n * length, 9)[: n * length]
    v[: 4 * length] = np.array(to_limbs(P - 1), np.uint64)
    got = poseidon2_hash_many(dev(v), length).cpu().numpy().view(np.uint64)
    for i in range(n):
        e = np.zeros(4, np.uint64)
        x = np.ascontiguousarray(v[i * length:(i + 1) * length])
        O.lib().pko_poseidon2_hash(O.p64(e), O.p64(x), length)
        assert np.array_equal(got[i], e), i
