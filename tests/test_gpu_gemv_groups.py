"""Request groups of the plain engine (one pass over the matrices for up to
four requests) against exact wrapping products, on both sides of the row
count at which a block takes four rows."""
import ctypes

import numpy as np
import pytest
import torch

from inspire_gb300 import _lib, pir, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("d,t", [(32, 1), (1024, 4), (1024, 8)])
def test_groups_match_exact_products(bits, d, t):
    p = synthetic.make_params(d=d, n=t * 136, t=t, coeff_bits=bits)
    m = synthetic.make_material(p, seed=d + t + bits)
    srv = pir.PirServer.CreateCombined(p, m.db, m.pack, m.a_tilde_agg,
                                       m.t_vec_h, m.second_dim_a)
    rows, kd = m.db.shape[0], m.pack.shape[1]
    view = np.int32 if bits == 32 else np.int64
    err = ctypes.create_string_buffer(256)
    for batch in range(1, 9):
        fd, _, pk = synthetic.make_requests(p, batch, seed=batch,
                                            full_range=True)
        yg = pk.reshape(batch, -1)[:, :kd]
        mod = np.uint64((1 << bits) - 1)
        want = (fd.astype(np.uint64) @ m.db.T.astype(np.uint64)
                + yg.astype(np.uint64)
                @ m.pack.T.astype(np.int64).astype(np.uint64)) & mod
        t_fd, t_pk = (torch.from_numpy(x.view(view)).cuda() for x in (fd, pk))
        out = torch.empty((batch, rows), device="cuda",
                          dtype=torch.int32 if bits == 32 else torch.int64)
        rc = _lib.load().inspire_pir_products_device(
            srv._h, batch, t_fd.data_ptr(), t_pk.data_ptr(), out.data_ptr(),
            pir.ENGINE_PLAIN, 0, err, len(err))
        assert rc == 0, err.value
        torch.cuda.synchronize()
        got = out.cpu().numpy().view(p.coeff_dtype).astype(np.uint64)
        assert np.array_equal(got, want), batch


@pytest.mark.parametrize("bits,db_dtype,mat_dtype", [
    (32, np.uint8, np.int32), (32, np.uint8, np.uint32),
    (64, np.uint16, np.uint64), (64, np.uint8, np.int32)])
@pytest.mark.parametrize("d,t,cols", [(64, 1, 1024), (1024, 8, 48),
                                      (1024, 8, 4096), (1024, 8, 8208)])
def test_rows_per_block_by_type_and_share(bits, db_dtype, mat_dtype, d, t,
                                          cols):
    # Few rows, and 8192 with the database below, at and above the shares of
    # the pack matrix at which a block of four requests takes four rows.
    p = synthetic.make_params(d=d, n=t * cols, t=t, coeff_bits=bits)
    rng = np.random.default_rng(cols + bits)
    rows, kd = d * t, 2 * d
    info = np.iinfo(mat_dtype)
    db = rng.integers(0, np.iinfo(db_dtype).max, (rows, cols), dtype=db_dtype,
                      endpoint=True)
    pack = rng.integers(info.min, info.max, (rows, kd), dtype=mat_dtype,
                        endpoint=True)
    zeros = np.zeros((2 * t + 6, d), p.coeff_dtype)
    srv = pir.PirServer.CreateCombined(p, db, pack, zeros[:t], zeros[:2 * t],
                                       zeros[:6] if t > 1 else None)
    view = np.int32 if bits == 32 else np.int64
    mod = np.uint64((1 << bits) - 1)
    some = np.unique(np.concatenate([np.arange(16), np.arange(rows - 16, rows),
                                     rng.integers(0, rows, 32)]))
    db64 = db[some].T.astype(np.uint64)
    pack64 = (pack[some].T.astype(np.int64) if info.min < 0
              else pack[some].T).astype(np.uint64)
    err = ctypes.create_string_buffer(256)
    for batch in (3, 4, 7):
        fd, _, pk = synthetic.make_requests(p, batch, seed=batch,
                                            first_dim_len=srv.db_cols,
                                            full_range=True)
        yg = pk.reshape(batch, -1)[:, :kd]
        want = (fd[:, :cols].astype(np.uint64) @ db64
                + yg.astype(np.uint64) @ pack64) & mod
        t_fd, t_pk = (torch.from_numpy(x.view(view)).cuda() for x in (fd, pk))
        out = torch.empty((batch, rows), device="cuda",
                          dtype=torch.int32 if bits == 32 else torch.int64)
        rc = _lib.load().inspire_pir_products_device(
            srv._h, batch, t_fd.data_ptr(), t_pk.data_ptr(), out.data_ptr(),
            pir.ENGINE_PLAIN, 0, err, len(err))
        assert rc == 0, err.value
        torch.cuda.synchronize()
        got = out.cpu().numpy().view(p.coeff_dtype).astype(np.uint64)
        assert np.array_equal(got[:, some], want), batch
