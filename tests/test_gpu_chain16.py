"""The cluster form of the reduction chains (d = 2048) against the oracle: one
digit, rounds of two with an odd one left, rounded gadgets, the widest digits
it takes and one above, which the block form runs."""
import numpy as np
import pytest

from inspire_gb300 import pir
from oracle import pyoracle as orc
from tests.rlwe_helpers import dtype_of, qmask

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,log_q,log_digit,k", [
    (32, 32, 20, 1), (32, 30, 9, 3), (64, 64, 16, 4), (64, 52, 27, 2),
    (32, 32, 28, 1)])
def test_matches_oracle(bits, log_q, log_digit, k):
    d = 2048
    rng = np.random.default_rng(100 * k + log_digit)
    mask = qmask(log_q, bits)
    hint = rng.integers(0, mask, (d, d), dtype=np.uint64,
                        endpoint=True).astype(dtype_of(bits))
    pack_a = rng.integers(0, mask, (2 * k, d), dtype=np.uint64,
                          endpoint=True).astype(dtype_of(bits))
    a, m, th = pir.PreprocessMatrixPack(hint, pack_a, log_q, log_digit, k)
    ref = orc.preprocess_matrix_pack(hint, pack_a[:k], pack_a[k:], bits,
                                     log_q, log_digit, k)
    assert np.array_equal(a[0], ref["a_tilde_agg"])
    assert np.array_equal(th[0], ref["t_vec_h"])
    assert np.array_equal(m, ref["matrix"].astype(dtype_of(bits)))
