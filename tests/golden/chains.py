"""PreprocessMatrixPack at ring degrees where the oracle takes minutes: seeded
inputs, and digests of the oracle's exact outputs for one slice of them.

  python tests/golden/chains.py [case ...]

computes the digests (chains.json beside this file).
"""
import hashlib
import json
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)
PATH = os.path.join(os.path.dirname(os.path.abspath(__file__)), "chains.json")

# name -> d, coefficient bits, log q, log digit, digits, slices, the slice that
# the digests are of, with the matrix
CASES = {
    "d2048_u64_q60_6x10": (2048, 64, 60, 6, 10, 1, 0, False),
    "d2048_u64_q64_45x1": (2048, 64, 64, 45, 1, 2, 1, True),
    "d4096_u32_q32_19x2": (4096, 32, 32, 19, 2, 2, 1, True),
    "d4096_u64_q52_19x2": (4096, 64, 52, 19, 2, 2, 1, False),
    "d4096_u32_q32_8x4": (4096, 32, 32, 8, 4, 2, 1, False),
    "d4096_u64_q52_14x3": (4096, 64, 52, 14, 3, 2, 1, False),
    "d8192_u32_q32_12x2": (8192, 32, 32, 12, 2, 1, 0, False),
    "d8192_u64_q64_30x1": (8192, 64, 64, 30, 1, 1, 0, False),
}


def words(seed, shape, log_q, dtype):
    """SplitMix64 of a counter, below 2^log_q."""
    n = int(np.prod(shape))
    with np.errstate(over="ignore"):
        z = (np.arange(1, n + 1, dtype=np.uint64)
             + np.uint64(seed << 40)) * np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z ^= z >> np.uint64(31)
    return (z >> np.uint64(64 - log_q)).astype(dtype).reshape(shape)


def inputs(name):
    """hint (slices d x d) and pack_a (2 k x d) of a case."""
    d, bits, log_q, _, k, slices, _, _ = CASES[name]
    dt = np.uint32 if bits == 32 else np.uint64
    seed = 1 + sorted(CASES).index(name)
    return (words(2 * seed, (slices * d, d), log_q, dt),
            words(2 * seed + 1, (2 * k, d), log_q, dt))


def digest(a):
    return hashlib.sha256(np.ascontiguousarray(a).tobytes()).hexdigest()


def make(name):
    from oracle import pyoracle as orc
    d, bits, log_q, log_digit, k, _, s, matrix = CASES[name]
    hint, pack_a = inputs(name)
    ref = orc.preprocess_matrix_pack(hint[s * d:(s + 1) * d], pack_a[:k],
                                     pack_a[k:], bits, log_q, log_digit, k,
                                     with_matrix=matrix)
    out = {"a_tilde_agg": digest(ref["a_tilde_agg"]),
           "t_vec_h": digest(ref["t_vec_h"])}
    if matrix:
        out["matrix"] = digest(ref["matrix"].astype(hint.dtype))
    return out


if __name__ == "__main__":
    for n in sys.argv[1:] or CASES:
        result = make(n)
        done = {}
        if os.path.exists(PATH):
            with open(PATH) as f:
                done = json.load(f)
        done[n] = result
        with open(PATH, "w") as f:
            json.dump(done, f, indent=1, sort_keys=True)
            f.write("\n")
