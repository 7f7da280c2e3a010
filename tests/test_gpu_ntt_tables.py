"""The device-built twiddle tables: products by a monomial are signed shifts,
at every ring degree (plain tables) and at the degrees of the radix-16
transforms (their permuted order)."""
import numpy as np
import pytest

from inspire_gb300 import pir

pytestmark = pytest.mark.gpu


def shift(v, e):
    """v * X^e mod X^d + 1 over Z_2^64."""
    d = v.size
    out = np.zeros_like(v)
    out[e:] = v[:d - e]
    out[:e] = 0 - v[d - e:]
    return out


@pytest.mark.parametrize("logd", range(1, 14))
def test_plain_tables(logd):
    d = 1 << logd
    rng = np.random.default_rng(logd)
    v = rng.integers(0, 1 << 64, d, dtype=np.uint64)
    for e in sorted({0, 1, d // 2, d - 1, int(rng.integers(d))}):
        u = np.zeros(d, np.uint64)
        u[e] = 1
        assert np.array_equal(pir.inner_product(u, v, 64), shift(v, e))


@pytest.mark.parametrize("logd", [11, 12, 13])
@pytest.mark.parametrize("n", [1, 3])
def test_permuted_tables(logd, n):
    """Row r of the database is a monomial in its last block: the hint row is
    the shift of that block's inverted a-component."""
    d = 1 << logd
    rng = np.random.default_rng(100 + logd)
    a = rng.integers(0, 1 << 64, (n, d), dtype=np.uint64)
    inv = np.concatenate([a[-1, :1], 0 - a[-1, :0:-1]])
    es = sorted({0, 1, d // 2, d - 1, int(rng.integers(d))})
    db = np.zeros((len(es), n * d), np.uint16)
    for r, e in enumerate(es):
        db[r, (n - 1) * d + e] = 65535
    got = pir.ComputeHintMatrix(db, a)
    for r, e in enumerate(es):
        assert np.array_equal(got[r], shift(inv, e) * np.uint64(65535))
