"""GPU parity of the tiled transform passes where their shapes change, word for
word against the oracle: fewer butterflies than a tile has threads, both tile
sizes, column counts that are no powers of two (lines cut at their power-of-two
part), skipped stages, the encode's loads in the first pass, and inputs at the
ends of the range (0, 1, p - 1) that drive the loosely reduced values to their
bounds."""
import numpy as np
import pytest
import torch

import oracle_lib as O
from fieldutil import P, to_limbs
from test_gpu_field import _lib  # noqa: F401
from provekit_b200.ntt import intt_rn, ntt_nr
from provekit_b200.rs import RSFr

pytestmark = pytest.mark.gpu


def values(n, seed, kind):
    edge = np.array([to_limbs(v) for v in (P - 1, 0, 1, P - 2)], np.uint64)
    if kind == "top":
        return np.repeat(edge[:1], n, axis=0)
    if kind == "edges":
        return edge[np.random.default_rng(seed).integers(0, 4, n)]
    return O.sample_fr(seed, n)


def dev(a):
    return torch.from_numpy(a.view(np.int64).copy()).cuda()


@pytest.mark.parametrize("kind", ["random", "edges", "top"])
@pytest.mark.parametrize("log_n,columns,groups", [
    (1, 1, 1), (2, 1, 1), (3, 5, 1), (7, 1, 1), (8, 1, 2), (9, 3, 1), (10, 1, 1), (11, 6, 4),
    (12, 12, 1), (16, 1, 1), (17, 1, 8)])
def test_forward(log_n, columns, groups, kind):
    n = 1 << log_n
    a = values(n * columns, log_n + columns, kind)
    got = ntt_nr(dev(a), n, groups).cpu().numpy().view(np.uint64)
    assert O.ntt_nr(a, n, groups) == 0
    assert np.array_equal(got, a)


@pytest.mark.parametrize("log_n", [20, 21])
def test_both_tile_sizes(log_n):
    n = 1 << log_n
    a = values(n, log_n, "edges")
    d = ntt_nr(dev(a), n, 1)
    exp = a.copy()
    assert O.ntt_nr(exp, n, 1) == 0
    assert np.array_equal(d.cpu().numpy().view(np.uint64), exp)
    assert np.array_equal(intt_rn(d).cpu().numpy().view(np.uint64), a)


@pytest.mark.parametrize("M,L,masks,log_cw", [(1, 2, 0, 2), (3, 5, 0, 4), (5, 100, 7, 8),
                                              (16, 1000, 0, 12), (12, 5003, 60, 15)])
def test_encode(M, L, masks, log_cw):
    m = values(M * L, M + L, "edges").reshape(M, L, 4)
    k = values(masks, 3, "random")
    rc, exp = O.rs_interleaved_encode(m, k, 1 << log_cw)
    assert rc == 0
    got = RSFr().interleaved_encode(dev(m), dev(k) if masks else None, 1 << log_cw)
    assert np.array_equal(got.cpu().numpy().view(np.uint64), exp)


@pytest.mark.parametrize("log_n", [1, 9, 10, 16, 17])
def test_inverse_of_both_grids(log_n):
    """Up to two CTAs of a pass per SM (2^16) and above."""
    a = values(1 << log_n, log_n, "edges")
    d = ntt_nr(dev(a), 1 << log_n, 1)
    assert np.array_equal(intt_rn(d).cpu().numpy().view(np.uint64), a)


@pytest.mark.parametrize("log_n,columns,groups", [(8, 3, 1), (9, 7, 1), (10, 7, 2), (10, 5, 4),
                                                  (13, 11, 1), (15, 12, 1), (17, 3, 1)])
def test_columns_that_cut_the_last_pass(log_n, columns, groups):
    """Odd column counts, whose last pass takes more stages than the passes before."""
    n = 1 << log_n
    a = values(n * columns, 5 + log_n, "edges")
    got = ntt_nr(dev(a), n, groups).cpu().numpy().view(np.uint64)
    assert O.ntt_nr(a, n, groups) == 0
    assert np.array_equal(got, a)
