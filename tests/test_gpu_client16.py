"""The client's radix-16 kernels against the definition of a sample: b = e - a s
plus the row's message, with the error's hash stream and the products redone
on the host (exact inner products of the oracle), and decryption against the
same arithmetic in Python integers."""
import numpy as np
import pytest

from inspire_gb300 import pir, synthetic
from oracle import pyoracle as orc

pytestmark = pytest.mark.gpu
M64 = (1 << 64) - 1


def mix(z):
    z = (z + np.uint64(0x9E3779B97F4A7C15))
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def errors(seed, ctr, var):
    """Centred binomials of the hash bits: 2 var bits minus 2 var bits."""
    n = 2 * var
    acc = np.zeros(ctr.size, np.int64)
    for word in range((2 * n + 63) // 64):
        bits = mix(np.uint64(seed) ^ mix((ctr << np.uint64(6))
                                         + np.uint64(word)))
        for i in range(64):
            at = 64 * word + i
            bit = ((bits >> np.uint64(i)) & np.uint64(1)).astype(np.int64)
            if at < n:
                acc += bit
            elif at < 2 * n:
                acc -= bit
    return acc


def times_key(a, s, bits):
    """a s over Z_2^bits."""
    v = s.astype(np.int64).astype(np.uint64)
    if bits == 32:
        v = v.astype(np.uint32)
    return orc.inner_product(a[None], v[None], bits, bits, bits, 20)


@pytest.mark.parametrize("d,t,bits,log_q,var", [
    (2048, 4, 32, 32, 40), (2048, 1, 64, 52, 6), (4096, 8, 32, 30, 16),
    (4096, 2, 64, 64, 33), (8192, 2, 32, 32, 40), (8192, 2, 64, 56, 40)])
def test_rows_and_decryption(d, t, bits, log_q, var):
    n = (d + 37) * t  # a ragged second first-dimension sample
    p = synthetic.make_params(d=d, n=n, t=t, coeff_bits=bits, log_q=log_q)
    cdt, k, ne = p.coeff_dtype, 2, 3 if t > 1 else 0
    rows = p.NumFirstDimSamples() + 2 * ne + 2 * k
    rng = np.random.default_rng(d + bits)
    a = rng.integers(0, 1 << log_q if log_q < 64 else M64, (rows, d),
                     dtype=np.uint64).astype(cdt)
    c = pir.PirClient.Create(p, a, clients=2, seed=5, variance=var)
    idx = np.array([n - 1, 3])
    fd, sd, pk = c.CreateRequests(idx, seed=77)
    mask = cdt(M64 >> (64 - log_q))
    for b in range(2):
        got = np.concatenate([fd[b], sd[b].reshape(-1), pk[b].reshape(-1)])
        want = []
        s = c.secret_keys[b]
        for row in range(rows):
            ctr = np.uint64((b * rows + row) * d) + np.arange(d,
                                                              dtype=np.uint64)
            e = errors(77, ctr, var).astype(np.uint64).astype(cdt)
            v = (e - times_key(a[row], s, bits)) & mask
            ns = p.NumFirstDimSamples()
            if row < ns:
                pos = int(idx[b]) // t - row * d
                if 0 <= pos < d:
                    hot = ((1 << log_q) + 65535 // 2) // 65535
                    v[pos] = (int(v[pos]) + hot) & int(mask)
                v = v[:fd.shape[1] - row * d]
            else:
                g = row - ns
                mono = (2 * d // t) * (int(idx[b]) % t)
                unit = np.zeros(d, np.int64)
                unit[mono % d] = -1 if mono >= d else 1
                if g < 2 * ne:
                    dig, ld, nd = g % ne, 19, ne
                    if g >= ne:
                        tgt = unit
                    else:
                        tgt = np.zeros(d, np.int64)
                        for j in range(d):
                            q = j + mono
                            tgt[q % d] = s[j] * (-1 if q // d % 2 else 1)
                else:
                    g -= 2 * ne
                    dig, ld, nd = g % k, 19, k
                    power = 5 if g < k else 2 * d - 1
                    q = np.arange(d) * power % (2 * d)
                    tgt = np.zeros(d, np.int64)
                    tgt[q % d] = np.where(q >= d, -s.astype(np.int64), s)
                sh = dig * ld + max(0, log_q - nd * ld)
                if sh < bits:
                    v = (v + (tgt.astype(np.uint64).astype(cdt) << cdt(sh))
                         ) & mask
            want.append(v)
        assert np.array_equal(got, np.concatenate(want)), b
    q1, q2 = (p.rlwe.log_modulus1_after_switch,
              p.rlwe.log_modulus2_after_switch)
    resp = rng.integers(0, M64, (2, 1, 2, d), dtype=np.uint64).astype(cdt)
    out = c.ProcessResponses(resp)
    for b in range(2):
        as_ = times_key(resp[b, 0, 0], c.secret_keys[b], bits)
        for j in list(range(0, d, 97)) + [d - 1]:
            x = int(as_[j]) & ((1 << q1) - 1)
            if q2 >= q1:
                x <<= q2 - q1
            else:
                x = (x >> (q1 - q2)) + ((x >> (q1 - q2 - 1)) & 1)
            v = (int(resp[b, 0, 1, j]) + x) & ((1 << q2) - 1)
            want = ((v * 65535 + (1 << q2) // 2) >> q2) % 65535
            assert int(out[b, j]) == want, (b, j)
