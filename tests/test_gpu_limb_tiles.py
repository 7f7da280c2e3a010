"""Request tiles of 16, 32, 48 and 64 in both forms of the tensor engine (the
raw form needs DB rows of a multiple of 16 bytes; batches above 64 use the
resident planes): batches at the edges of every tile against the plain
engine, untuned and tuned, with operands at the ends of the digits' range."""
import ctypes

import numpy as np
import pytest
import torch

from inspire_gb300 import _lib, pir, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [392, 389])
def test_tiles_match_plain_engine(cols):
    p = synthetic.make_params(d=256, n=4 * cols, t=4, coeff_bits=32)
    m = synthetic.make_material(p, seed=cols)
    db = m.db.copy()
    db[:256] = 65535
    db[256:512] = 0
    srv = pir.PirServer.CreateCombined(p, db, m.pack, m.a_tilde_agg,
                                       m.t_vec_h, m.second_dim_a)
    lib, err = _lib.load(), ctypes.create_string_buffer(256)
    for batch in (1, 16, 17, 31, 32, 33, 45, 48, 49, 64, 65, 96, 97, 130):
        fd, _, pk = synthetic.make_requests(p, batch, seed=batch,
                                            full_range=True)
        fd[0] = 0x80808080  # every balanced digit at -128
        fd[-1] = 0x7F7F7F7F
        t_fd, t_pk = (torch.from_numpy(x.view(np.int32)).cuda()
                      for x in (fd, pk))
        outs = []
        for engine in (pir.ENGINE_PLAIN, pir.ENGINE_TENSOR, pir.ENGINE_TENSOR):
            out = torch.full((batch, db.shape[0]), -1, dtype=torch.int32,
                             device="cuda")
            rc = lib.inspire_pir_products_device(
                srv._h, batch, t_fd.data_ptr(), t_pk.data_ptr(),
                out.data_ptr(), engine, 0, err, len(err))
            assert rc == 0, err.value
            torch.cuda.synchronize()
            outs.append(out)
            if len(outs) == 2:
                srv.autotune(batch)
        srv.check()
        assert torch.equal(outs[0], outs[1]), batch
        assert torch.equal(outs[0], outs[2]), batch
