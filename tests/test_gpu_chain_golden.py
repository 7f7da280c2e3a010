"""PreprocessMatrixPack word for word at d = 4096 and at other rings whose
oracle run takes minutes: digests of the oracle's exact outputs, computed once
(tests/golden/chains.py). Two slices where the digest is of the second: the
blocks' slice offsets count too. Cases: the cluster chains of d = 4096 for both
word sizes, the largest digit counts that the register links take, digits
wider than a prime."""
import json

import numpy as np
import pytest

from inspire_gb300 import pir
from tests.golden import chains

pytestmark = pytest.mark.gpu


def check(name):
    d, _, log_q, log_digit, k, _, s, _ = chains.CASES[name]
    with open(chains.PATH) as f:
        want = json.load(f)[name]
    hint, pack_a = chains.inputs(name)
    a, m, th = pir.PreprocessMatrixPack(hint, pack_a, log_q, log_digit, k)
    assert chains.digest(a[s]) == want["a_tilde_agg"]
    assert chains.digest(th[s]) == want["t_vec_h"]
    if "matrix" in want:
        assert chains.digest(m[s * d:(s + 1) * d]) == want["matrix"]


@pytest.mark.parametrize("name", [
    "d4096_u32_q32_19x2", "d4096_u64_q52_19x2", "d4096_u64_q52_14x3",
    "d4096_u32_q32_8x4", "d2048_u64_q60_6x10", "d2048_u64_q64_45x1"])
def test_matches_oracle_digests(name):
    check(name)


def test_digest_sees_one_word():
    x = np.arange(8, dtype=np.uint64)
    y = x.copy()
    y[3] ^= np.uint64(1)
    assert chains.digest(x) != chains.digest(y)


@pytest.mark.parametrize("name", ["d8192_u64_q64_30x1"])
def test_general_chains_of_wide_rings(name):
    # Digits of 29 bits and more over Z_2^64: four 31-bit primes fit, five
    # 27-bit ones do not.
    check(name)


@pytest.mark.parametrize("name", ["d8192_u32_q32_12x2"])
def test_cluster_chains_at_d8192(name):
    # Twiddles and key parts from global memory.
    check(name)
