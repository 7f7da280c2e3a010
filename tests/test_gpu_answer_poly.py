"""The one-launch polynomial stage (d = 2048, 4096) against the oracle: word
sizes, moduli below and at the word size (the last slice's own inverse
transform), slice counts from one, shards, gadgets of one digit per group and
of several rounds, and gadgets it leaves to the launch-per-step kernels."""
import numpy as np
import pytest

from inspire_gb300 import pir, synthetic
from oracle import pyoracle as orc

pytestmark = pytest.mark.gpu

CASES = [  # d, t, l, bits, log_q, pack gadget, eval gadget, batch
    (2048, 1, 1, 32, 32, (19, 2), (19, 3), 1),
    (2048, 2, 2, 32, 30, (19, 2), (19, 3), 3),
    (2048, 4, 1, 32, 32, (8, 4), (8, 4), 2),      # eight digits: two rounds
    (2048, 2, 1, 32, 32, (19, 2), (2, 16), 1),    # 32 digits: not fused
    (2048, 1, 2, 64, 52, (19, 2), (19, 3), 2),
    (2048, 4, 1, 64, 64, (19, 2), (19, 3), 1),    # eight digits of six groups
    (2048, 2, 2, 64, 56, (19, 2), (19, 3), 3),
    (4096, 2, 1, 32, 32, (19, 2), (19, 3), 2),
    (4096, 4, 2, 32, 31, (19, 2), (10, 3), 1),    # GadgetInv rounds a bit off
    (4096, 1, 1, 64, 52, (19, 2), (19, 3), 1),
    (4096, 2, 1, 64, 52, (19, 2), (19, 3), 2),
    (4096, 2, 1, 64, 64, (19, 2), (28, 2), 1),    # digits above the primes
]


@pytest.mark.parametrize("case", CASES, ids=[str(c) for c in CASES])
def test_matches_oracle(case):
    d, t, l, bits, log_q, pack, evalg, batch = case
    p = synthetic.make_params(d=d, n=64 * t, t=t, l=l, coeff_bits=bits,
                              log_q=log_q, pack=pack, evalg=evalg)
    m = synthetic.make_material(p, seed=d + t + bits, db_cols=64)
    srv = pir.PirServer.CreateCombined(p, m.db, m.pack, m.a_tilde_agg,
                                       m.t_vec_h, m.second_dim_a)
    fd, sd, pk = synthetic.make_requests(p, batch, seed=log_q,
                                         full_range=True)
    got = srv.process_arrays(fd, sd, pk)
    r = p.rlwe
    op = orc.make_params(
        coeff_bits=bits, log_degree=d.bit_length() - 1, log_modulus=log_q,
        log_modulus1_after_switch=r.log_modulus1_after_switch,
        log_modulus2_after_switch=r.log_modulus2_after_switch,
        pack_log_digit=pack[0], pack_num_digits=pack[1],
        eval_log_digit=evalg[0], eval_num_digits=evalg[1],
        num_entries=64 * t, interpolation_degree=t, entry_size_multiple=l)
    for i in range(batch):
        want = orc.process_response(op, m.db, m.pack, m.a_tilde_agg,
                                    m.t_vec_h, m.second_dim_a, fd[i], sd[i],
                                    pk[i])
        assert np.array_equal(got[i], want), i


@pytest.mark.parametrize("case", [
    # One digit of 30 bits, above the 27-bit primes, in the one launch.
    (2048, 2, 1, 32, 32, (19, 2), (30, 1), 2),
    (4096, 4, 1, 32, 32, (19, 2), (29, 1), 2),
    # Eight live digits on six groups: a second round of two.
    (2048, 4, 1, 64, 64, (19, 2), (16, 4), 2),
    (2048, 2, 2, 64, 52, (19, 2), (13, 4), 1),
    # d = 4096 over Z_2^64: eight live digits on three groups.
    (4096, 2, 1, 64, 64, (19, 2), (16, 4), 1),
], ids=str)
def test_wide_digits_and_second_rounds(case):
    test_matches_oracle(case)
