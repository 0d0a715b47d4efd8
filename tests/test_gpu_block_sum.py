"""The block-wide limb sums behind pkg_dot at their bounds, against Python
integers: every thread of every CTA contributing p - 1 (the largest limbs, the
most carries), one CTA (which skips the ticket), one thread more, and the last
CTA of a full grid nearly empty."""
import numpy as np
import pytest
import torch

from fieldutil import P, from_limbs, to_limbs
from test_gpu_field import _lib  # noqa: F401
from provekit_b200.spartan import dot

pytestmark = pytest.mark.gpu

R = 1 << 256
RINV = pow(2, -256, P)


@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 256, 257, 65536, 151553])
@pytest.mark.parametrize("value", [P - 1, R % P, 1])
def test_equal_terms(n, value):
    a = torch.from_numpy(np.tile(np.array(to_limbs(value), np.uint64), (n, 1)).view(np.int64)).cuda()
    one = torch.from_numpy(np.tile(np.array(to_limbs(R % P), np.uint64), (n, 1)).view(np.int64)).cuda()
    assert from_limbs(dot(a, one)) == n * value % P
    assert from_limbs(dot(a, a)) == n * value * value * RINV % P
