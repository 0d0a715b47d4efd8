"""GPU parity of the unreduced product sums at the edges of their splits: the
points of an equality sum shared by 1, 2, 4 and 8 threads, more than 1024 terms
per thread, tables shorter than a CTA; and sums whose operands are all p - 1 (the
largest words and the most carries)."""
import numpy as np
import pytest
import torch

import oracle_lib as O
from fieldutil import P, to_limbs
from test_gpu_field import _lib  # noqa: F401
from provekit_b200.spartan import dot
from provekit_b200.whir import eq_accumulate, fold_coeffs

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int64)).cuda()


@pytest.mark.parametrize("nv,npts", [(0, 1), (0, 8 * 1024 + 9), (1, 15), (1, 16), (2, 31), (5, 32),
                                     (8, 63), (9, 64), (9, 65), (14, 33), (16, 70)])
def test_eq_accumulate_splits(nv, npts):
    w = O.sample_fr(nv, 1 << nv)
    pts, cf = O.sample_fr(3 + nv, max(npts * nv, 1)), O.sample_fr(npts, npts)
    dw = dev(w)
    eq_accumulate(dw, nv, pts, cf)
    assert O.lib().pko_eq_accumulate(O.p64(w), nv, O.p64(pts), O.p64(cf), npts) == 0
    assert np.array_equal(dw.cpu().numpy().view(np.uint64), w)


@pytest.mark.parametrize("n", [1, 255, 257, 148 * 3 * 256 + 1])
def test_dot_of_largest_values(n):
    a = np.broadcast_to(np.array(to_limbs(P - 1), np.uint64), (n, 4)).copy()
    exp = to_limbs(n * (P - 1) ** 2 * pow(2, -256, P) % P)
    assert np.array_equal(dot(dev(a), dev(a)), np.array(exp, np.uint64))


@pytest.mark.parametrize("k", [0, 1, 6])
def test_fold_of_largest_values(k):
    c = np.broadcast_to(np.array(to_limbs(P - 1), np.uint64), (256 << k, 4)).copy()
    alpha = np.broadcast_to(np.array(to_limbs(P - 1), np.uint64), (max(k, 1), 4)).copy()
    got = fold_coeffs(dev(c), k, alpha).cpu().numpy().view(np.uint64)
    assert np.array_equal(got.reshape(-1, 4), O.whir_fold_coeffs(c, k, alpha))


@pytest.mark.parametrize("nv,npts", [(0, 3), (1, 2), (2, 5), (3, 1), (7, 9), (12, 3), (19, 2)])
def test_equality_tables(nv, npts):
    """Halves of every length from none, points as coordinates (a proof's univariate
    points are expanded in the same kernel: whole proofs)."""
    w = O.sample_fr(70 + nv, 1 << nv)
    pts, cf = O.sample_fr(71 + nv, max(npts * nv, 1)), O.sample_fr(72, npts)
    pts[0] = np.array(to_limbs(P - 1), np.uint64)
    dw = dev(w)
    eq_accumulate(dw, nv, pts, cf)
    assert O.lib().pko_eq_accumulate(O.p64(w), nv, O.p64(pts), O.p64(cf), npts) == 0
    assert np.array_equal(dw.cpu().numpy().view(np.uint64), w)


@pytest.mark.parametrize("nr,entries", [(0, 1), (3, 5), (8, 256), (9, 257), (9, 512), (14, 1 << 14),
                                        (18, (1 << 18) - 1), (19, 1 << 19), (25, (1 << 25) - 300)])
def test_equality_table_runs(nr, entries):
    """Fewer variables than a run's eight, runs cut short, one and several runs a CTA, and
    as many as a CTA takes (2^25 entries)."""
    from provekit_b200.spartan import eq_hypercube
    r = O.sample_fr(40 + nr, max(nr, 1))[:nr]
    if nr:
        r[-1] = np.array(to_limbs(P - 1), np.uint64)
    exp = np.zeros((entries, 4), np.uint64)
    assert O.lib().pko_eq_hypercube(O.p64(r) if nr else None, nr, entries, O.p64(exp)) == 0
    got = eq_hypercube(r, entries).cpu().numpy().view(np.uint64)
    assert np.array_equal(got, exp)
