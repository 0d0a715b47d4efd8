"""GPU parity of transforms of few stages over column counts that are no powers of two,
whose lines do not share their twiddles within a tile: one to eight stages, few and
many CTAs, the last lines of a group in one tile with the first of the next, and
encodes whose first coset is short, word for word against the oracle."""
import numpy as np
import pytest

import oracle_lib as O
from test_gpu_field import _lib  # noqa: F401
from test_gpu_ntt_tiles import dev, values
from provekit_b200.ntt import ntt_nr
from provekit_b200.rs import RSFr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_n,columns,stages", [
    (2, 3, 1), (5, 7, 2), (12, 33, 1), (12, 33, 2), (12, 6, 3), (13, 12, 5), (11, 5, 6), (12, 3, 7),
    (12, 3, 8), (14, 33, 1), (13, 257, 4), (15, 6, 7), (17, 7, 6), (18, 11, 2)])
def test_last_stages(log_n, columns, stages):
    n, groups = 1 << log_n, 1 << (log_n - stages)
    a = values(n * columns, 3 * log_n + stages, "edges" if log_n < 17 else "random")
    got = ntt_nr(dev(a), n, groups).cpu().numpy().view(np.uint64)
    assert O.ntt_nr(a, n, groups) == 0
    assert np.array_equal(got, a)


@pytest.mark.parametrize("M,L,masks,log_cw", [(5, 2, 0, 10), (3, 4, 3, 12), (11, 7, 0, 9), (6, 30, 9, 13)])
def test_encode_of_short_messages(M, L, masks, log_cw):
    m = values(M * L, M + L, "edges").reshape(M, L, 4)
    k = values(masks, 3, "random")
    rc, exp = O.rs_interleaved_encode(m, k, 1 << log_cw)
    assert rc == 0
    got = RSFr().interleaved_encode(dev(m), dev(k) if masks else None, 1 << log_cw)
    assert np.array_equal(got.cpu().numpy().view(np.uint64), exp)
