"""The hint rows of the radix-16 rings: every element type, one block, the
blocks around the fold of the 64-bit sums, and operands at the ends of their
range (the sums' and the reconstruction's bounds), against the oracle's exact
inner products."""
import numpy as np
import pytest

from inspire_gb300 import pir
from oracle import pyoracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n", [(2048, 1), (2048, 24), (2048, 49), (4096, 1),
                                 (4096, 25), (8192, 1), (8192, 25)])
@pytest.mark.parametrize("sdt,tdt", [(np.uint8, np.uint32),
                                     (np.uint16, np.uint32),
                                     (np.uint32, np.uint32),
                                     (np.uint8, np.uint64),
                                     (np.uint16, np.uint64),
                                     (np.uint32, np.uint64)])
def test_rows(d, n, sdt, tdt):
    rng = np.random.default_rng(d + n)
    smax, tmax = np.iinfo(sdt).max, np.iinfo(tdt).max
    db = rng.integers(0, smax, size=(4, d * n), dtype=sdt, endpoint=True)
    db[1] = smax
    db[2] = 0
    a = rng.integers(0, tmax, size=(n, d), dtype=tdt, endpoint=True)
    if n == 24:
        a[:] = tmax
    got = pir.ComputeHintMatrix(db, a)
    bits = 8 * np.dtype(tdt).itemsize
    vinv = np.concatenate([a[:, :1], (0 - a[:, :0:-1]).astype(tdt)], axis=1)
    chunk = min(20, int((53.0 - np.log2(n) - np.log2(d)) / 2.0))
    for i in range(db.shape[0]):
        want = orc.inner_product(db[i].reshape(n, d).astype(tdt), vinv, bits,
                                 8 * np.dtype(sdt).itemsize, bits, chunk)
        assert np.array_equal(got[i], want), i
