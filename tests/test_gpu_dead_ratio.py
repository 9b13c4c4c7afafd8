"""The fire pass's ratio of dead fuel moisture (csrc/fire.cu, dead_ratio): a
product with the reciprocal of the model's moisture of extinction, against the
quotient in double precision and against CUDA's __fdividef.

Bounds: CUDA states 2 units in the last place (at most 2^-22 of the value) for
__fdividef with a divisor in [2^-126, 2^126], which gives the reciprocal; the
product rounds once, 2^-24.  So the product lies within 2^-22 + 2^-24 of the
quotient, up to terms of 2^-46, and within 2^-22 more of __fdividef's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_dead_ratio(pp):
    from py_propag import _lib as L
    rng = np.random.default_rng(47)
    n = 1_300_000
    model = np.repeat(np.arange(1, 14, dtype=np.int32), n // 13)
    dead = rng.uniform(0.0, 0.4, n).astype(np.float32)
    dead[::7] = (0.4 * 2.0 ** rng.uniform(-24, 0, dead[::7].size)).astype(np.float32)
    product, quotient, mext = (np.zeros(n, np.float32) for _ in range(3))
    rc = L.lib().propag_selftest_dead_ratio(n, *[a.ctypes.data for a in (model, dead, product, quotient, mext)])
    assert rc == 0, L.last_error()
    assert np.all((mext > 0.05) & (mext < 0.5))
    exact = dead.astype(np.float64) / mext.astype(np.float64)
    bound = (2.0 ** -22 + 2.0 ** -24 + 2.0 ** -45) * exact
    assert np.all(np.abs(product.astype(np.float64) - exact) <= bound)
    assert np.all(np.abs(product.astype(np.float64) - quotient.astype(np.float64)) <= bound + 2.0 ** -22 * exact)
    print("largest distance from the quotient in 2^-24:", (np.abs(product / exact - 1) * 2 ** 24).max(),
          "; values other than __fdividef's:", np.mean(product != quotient))
