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


@pytest.mark.parametrize("omega", [0.5, 0.66, 0.81, 1.0])
@pytest.mark.parametrize("low,high", [(0.8, 1.3), (1e-6, 1e6)])
def test_relax_rate(cuda, omega, low, high):
    """1 / tau of density 1 is lambda^(omega - 1): pow is within 2 ulp over its range
    (CUDA's table), the products are by 1, and the reciprocal adds half an ulp; an ulp
    is at most 2^-52 of its value, and the host's power is good to 2^-60."""
    rng = np.random.default_rng(11)
    lam = np.exp(rng.uniform(np.log(low), np.log(high), 1 << 20))
    d = _lib.BlockDesc()
    d.relax_type, d.Kn_eff, d.omega, d.PI = 2, 1.0, omega, np.pi
    t = torch.from_numpy(lam).cuda()
    out = torch.empty_like(t)
    _lib.check(_lib.lib().ugks_check_relax_rate(C.byref(d), t.data_ptr(), len(lam), out.data_ptr(), stream()),
               "ugks_check_relax_rate")
    want = np.power(lam.astype(np.longdouble), -np.longdouble(1.0 - omega))
    err = np.abs(out.cpu().numpy().astype(np.longdouble) - want) / want
    assert np.max(err) <= 2.5 * 2.0 ** -52 + 2.0 ** -60
