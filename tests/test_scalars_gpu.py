"""The scalar functions of the face and cell coefficients against 64-bit-mantissa
values on the host."""
import ctypes as C

import numpy as np
import pytest
import torch

from pyugks_b200 import _lib

pytestmark = pytest.mark.gpu


def stream():
    return torch.cuda.current_stream().cuda_stream


def reciprocals(x):
    t = torch.from_numpy(x).cuda()
    y = torch.empty_like(t)
    _lib.check(_lib.lib().ugks_check_reciprocal(t.data_ptr(), len(x), y.data_ptr(), stream()), "ugks_check_reciprocal")
    return y.cpu().numpy()


@pytest.mark.parametrize("low", [0, 1, 2 ** 31, 2 ** 32 - 1, None])
def test_reciprocal(cuda, low):
    """Every value of the 20 mantissa bits that the approximate instruction reads, at
    the edges of what it cuts off and between them, over the exponents.  Two Newton
    steps leave (2^-19)^4 beside the last rounding, and the host's 1 / x 2^-64: half
    an ulp and 2^-10 of one."""
    rng = np.random.default_rng(7)
    n = 1 << 20
    high = np.arange(n, dtype=np.uint64) << np.uint64(32)
    bits = high | (rng.integers(0, 1 << 32, n, dtype=np.uint64) if low is None else np.uint64(low))
    exps = rng.integers(1023 - 900, 1023 + 900, n).astype(np.uint64) << np.uint64(52)
    sign = rng.integers(0, 2, n).astype(np.uint64) << np.uint64(63)
    for e in (np.uint64(1023) << np.uint64(52), exps | sign):
        x = (bits | e).view(np.float64)
        y = reciprocals(x)
        err = np.abs(y.astype(np.longdouble) - np.longdouble(1.0) / x.astype(np.longdouble))
        assert np.max(err / np.abs(np.spacing(y))) <= 0.5 + 2.0 ** -10
