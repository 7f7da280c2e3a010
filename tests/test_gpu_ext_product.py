"""The one-launch batched external product against the oracle: a group per
digit and digits in turns, rounding gadgets, digits above the primes, in
place, and a gadget whose range it leaves to the launch-per-stage kernels."""
import numpy as np
import pytest
import torch

from inspire_gb300 import pir, synthetic
from oracle import pyoracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,bits,log_q,evalg,batch", [
    (2048, 32, 32, (19, 3), 3), (2048, 32, 30, (8, 4), 2),
    (2048, 32, 32, (2, 16), 2), (2048, 64, 36, (18, 2), 2),
    (2048, 64, 52, (19, 3), 3), (2048, 64, 64, (28, 2), 1),
    (2048, 64, 64, (60, 1), 1), (4096, 32, 32, (19, 3), 2),
    (4096, 32, 31, (10, 3), 2), (4096, 64, 64, (19, 3), 2)])
def test_matches_oracle(d, bits, log_q, evalg, batch):
    p = synthetic.make_params(d=d, n=64, t=1, coeff_bits=bits, log_q=log_q,
                              evalg=evalg)
    m = synthetic.make_material(p, seed=d + bits, db_cols=64)
    srv = pir.PirServer.CreateCombined(p, m.db, m.pack, m.a_tilde_agg,
                                       m.t_vec_h, None)
    rng = np.random.default_rng(d + log_q)
    cdt, ne = p.coeff_dtype, evalg[1]
    top = np.iinfo(cdt).max
    ct = rng.integers(0, top, (batch, 2, d), dtype=cdt, endpoint=True)
    rgsw = rng.integers(0, top, (batch, 2 * ne, 2, d), dtype=cdt,
                        endpoint=True)
    ct[0, 0] = top
    rgsw[0] = top
    view = np.int32 if bits == 32 else np.int64
    t_ct, t_rg = (torch.from_numpy(x.view(view)).cuda() for x in (ct, rgsw))
    srv.external_product_device(batch, t_ct.data_ptr(), t_rg.data_ptr(),
                                t_ct.data_ptr())  # in place
    torch.cuda.synchronize()
    got = t_ct.cpu().numpy().view(cdt)
    r = p.rlwe
    op = orc.make_params(
        coeff_bits=bits, log_degree=d.bit_length() - 1, log_modulus=log_q,
        log_modulus1_after_switch=r.log_modulus1_after_switch,
        log_modulus2_after_switch=r.log_modulus2_after_switch,
        pack_log_digit=19, pack_num_digits=2, eval_log_digit=evalg[0],
        eval_num_digits=ne, num_entries=64, interpolation_degree=1,
        entry_size_multiple=1)
    for i in range(batch):
        wa, wb = orc.external_product(op, ct[i, 0], ct[i, 1],
                                      rgsw[i].reshape(-1, d))
        assert np.array_equal(got[i, 0], wa), i
        assert np.array_equal(got[i, 1], wb), i


@pytest.mark.parametrize("evalg", [(40, 1), (32, 2)])
def test_one_slice_server_with_wide_digits(evalg):
    # Products of 116 and 109 bits: five 27-bit primes, where the answers of
    # the same server take four.
    test_matches_oracle(2048, 64, 64, evalg, 2)


@pytest.mark.parametrize("d,evalg", [(2048, (4, 6)), (2048, (4, 7)),
                                     (4096, (2, 6)), (4096, (2, 16))])
def test_narrow_digits_on_either_side_of_the_one_launch_form(d, evalg):
    # Products of at most 51 bits: two primes where the one launch takes three.
    test_matches_oracle(d, 32, 32, evalg, 3)
