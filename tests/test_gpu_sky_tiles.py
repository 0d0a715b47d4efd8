"""GPU parity of the tiled Skyscraper folds and subtrees (128 compressions at a
time) at the edges of their tiles and of the rules that choose them, byte for
byte against the oracle: one message, a tile less one, a tile, one more, and a
count that gives some CTAs a second, partly filled tile; inputs of all ones
(not reduced), zero and p among random ones."""
import numpy as np
import pytest
import torch

import oracle_lib as O
from fieldutil import P, to_limbs
from test_gpu_field import _lib  # noqa: F401
from provekit_b200._lib import PKG_LEAF_CANONICAL, PKG_LEAF_MONTGOMERY
from provekit_b200.merkle import merkle_tree, merkle_tree_fr
from provekit_b200.skyscraper import SkyscraperHashEngine, compress_many

pytestmark = pytest.mark.gpu


def chunks(n, seed):
    v = np.random.default_rng(seed).integers(0, 2**64, (n, 4), dtype=np.uint64)
    edge = [(1 << 256) - 1, 0, P, P - 1, 2 * P, 1]
    for i, e in enumerate(edge[:n]):
        v[i] = to_limbs(e)
        v[n - 1 - i] = to_limbs(edge[-1 - i])
    return v


def dev_bytes(v):
    return torch.from_numpy(v.view(np.uint8).reshape(-1).copy()).cuda()


@pytest.mark.parametrize("count,size", [(1, 96), (1, 544), (127, 96), (128, 128), (129, 96),
                                        (151553, 96)])
def test_hash_many(count, size):
    v = chunks(count * size // 32, count + size)
    got = SkyscraperHashEngine().hash_many(size, dev_bytes(v)).cpu().numpy().tobytes()
    assert got == O.hash_many(size, v.tobytes(), count)


@pytest.mark.parametrize("count", [1, 1 << 15, (1 << 15) + 1, 151681])
def test_compress_many(count):
    v = chunks(2 * count, count)
    got = compress_many(dev_bytes(v)).cpu().numpy().tobytes()
    assert got == O.hash_many(64, v.tobytes(), count)


@pytest.mark.parametrize("encoding", [PKG_LEAF_CANONICAL, PKG_LEAF_MONTGOMERY])
@pytest.mark.parametrize("count,row", [(1, 3), (4, 1), (4, 2), (128, 5), (256, 8), (1 << 17, 2)])
def test_codeword_rows(encoding, count, row):
    v = chunks(count * row, 7 * count + row)
    v[:, 3] %= np.uint64(0x30644E72E131A029)
    cw = torch.from_numpy(v.view(np.int64).copy()).cuda()
    got = merkle_tree_fr(cw, row, encoding).cpu().numpy().tobytes()
    leaves = v.copy()
    if encoding == PKG_LEAF_CANONICAL:
        O.lib().pko_from_mont_many(O.p64(leaves), leaves.shape[0])
    assert got == O.merkle_tree(leaves.tobytes(), 32 * row, count)


@pytest.mark.parametrize("log_n", [0, 1, 5, 6, 7, 8, 9, 15, 16, 17])
def test_subtrees(log_n):
    v = chunks(1 << log_n, 100 + log_n)
    got = merkle_tree(dev_bytes(v), 32).cpu().numpy().tobytes()
    assert got == O.merkle_tree(v.tobytes(), 32, 1 << log_n)
