"""GPU parity of the integer-pipe products over their whole input range: the
kernels multiply operands up to 2p, so the two-accumulator rows and the
square's carry chains are checked at words of all ones and all zeros (every
carry taken, or none), at 2p - 1 and at random, against Python integers."""
import random

import pytest

from fieldutil import P
from test_gpu_field import _lib, dev, ints  # noqa: F401
from provekit_b200.field import fr_op

pytestmark = pytest.mark.gpu

RINV = pow(2, -256, P)
W = 0xFFFFFFFF


def values(bound, n, seed):
    rnd = random.Random(seed)
    v = [0, 1, P - 1, bound - 1, bound - 2]
    v += [W << (32 * i) for i in range(8)]
    v += [(1 << (32 * i)) - 1 for i in range(1, 9)]
    v += [sum(W << (32 * i) for i in range(p, 8, 2)) for p in (0, 1)]
    v += [sum(rnd.choice([0, 1, W - 1, W]) << (32 * i) for i in range(8)) for _ in range(300)]
    v = [x % bound for x in v] + [rnd.randrange(bound) for _ in range(n)]
    return v


@pytest.mark.parametrize("n", [1, 700])
def test_products_below_2p(n):
    a = values(2 * P, n, 11)
    b = values(2 * P, n, 12)
    random.Random(13).shuffle(b)
    assert ints(fr_op("mul", dev(a), dev(b), pipe="int")) == [x * y * RINV % P
                                                             for x, y in zip(a, b)]
    assert ints(fr_op("sqr", dev(a), pipe="int")) == [x * x * RINV % P for x in a]


def test_reduction_of_any_256_bits():
    a = values(1 << 256, 700, 14) + [(1 << 256) - 1]
    assert ints(fr_op("from_mont", dev(a), pipe="int")) == [x * RINV % P for x in a]
