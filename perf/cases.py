"""The work users of this framework have it do, as measurable cases.

Kinds of case:
  answer    ProcessResponse of device-resident requests on a device-resident
            server (process_device, INSPIRE_ENGINE_AUTO)
  host      ProcessBatch-style calls with host arrays (process_arrays)
  vpir      the vPIR server's answer, host arrays
  pack      the packing tool's server step and one external product per
            instance, device-resident
  client    request creation and response decryption of a batch of clients,
            device-resident
  interp    offline: interpolation and transposition of a raw database
  hint      offline: the hint matrix of a database
  material  offline: PreprocessMatrixPack of a hint matrix

Every output is a whole number (ring elements, database words), held bit for
bit; there is no floating output, so no 64-bit floating reference either.
"""
import ctypes
import math

import numpy as np
import torch

from inspire_gb300 import _lib, pir, synthetic

# Modulus and gadgets per word size: Z_2^32 with q = 2^32 and a 19 x 3 eval
# gadget; Z_2^64 with the reference's q = 2^52 and 2^56.
U16_MAX = 65535


def listed():
    return [
        # One request on the reference metrics tool's default database, the
        # smallest call: launches and latency.
        dict(name="answer_metrics_tool_b1", kind="answer", n=4096, d=2048,
             t=2, l=1, bits=64, log_q=52, batch=1),
        # One request through the reference-like call with host arrays, on
        # the metrics tool's small-database shape.
        dict(name="host_n65536_b1", kind="host", n=65536, d=2048, t=4, l=1,
             bits=32, log_q=32, batch=1),
        # Serving at light load, the large ring: a few requests that share
        # one pass over a 4 GiB database with two-polynomial records.
        dict(name="answer_ring8192_b3", kind="answer", n=131072, d=8192, t=2,
             l=2, bits=32, log_q=32, batch=3),
        # Serving at moderate load: a small batch on a quarter of the
        # benchmarked database.
        dict(name="answer_n262144_b12", kind="answer", n=262144, d=4096, t=8,
             l=1, bits=32, log_q=32, batch=12),
        # A ragged batch on a ragged record count (columns are no multiple
        # of the ring degree).
        dict(name="answer_n200000_b45", kind="answer", n=200000, d=4096, t=8,
             l=1, bits=32, log_q=32, batch=45),
        # The reference's 64-bit parameters in a batch.
        dict(name="answer_u64_n131072_b96", kind="answer", n=131072, d=2048,
             t=8, l=1, bits=64, log_q=56, batch=96),
        # The headline benchmark: 2^20 records, 256 requests.
        dict(name="answer_n1048576_b256", kind="answer", n=1048576, d=4096,
             t=8, l=1, bits=32, log_q=32, batch=256),
        # The packing micro-workload: LWE-to-RLWE packing of one ring
        # element per instance and an external product each.
        dict(name="pack_d2048_b256", kind="pack", n=2048, d=2048, t=1, l=1,
             bits=32, log_q=32, batch=256),
        # Load generation: requests for and decryption of a batch of
        # answers (encode and decode).
        dict(name="client_n262144_b64", kind="client", n=262144, d=4096, t=8,
             l=1, bits=32, log_q=32, batch=64),
        # Offline: a raw database to its interpolated, transposed form.
        dict(name="interp_n131072", kind="interp", n=131072, d=4096, t=8,
             l=1, value_bits=16),
        # Offline: the hint matrix of a small database.
        dict(name="hint_n262144", kind="hint", n=262144, d=4096, t=8, l=1,
             bits=32),
        # Offline: the packing material of eight slices under the metrics
        # tool's ring and modulus.
        dict(name="material_d2048_s8", kind="material", d=2048, slices=8,
             bits=64, log_q=52),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["answer", "answer", "answer", "host", "vpir", "pack",
                       "client", "interp", "hint", "material"])
    bits = rng.choice([32, 32, 64])
    log_q = 32 if bits == 32 else rng.choice([52, 56])
    ring = rng.choice([(2048, 2), (2048, 4), (2048, 8), (4096, 8), (4096, 4),
                       (8192, 2)])
    d, t = ring
    l = rng.choice([1, 1, 1, 2])
    if kind == "answer":
        # Up to 4 GiB of database; the largest batches on the smaller ones.
        cols = _log_int(rng, 512, (1 << 31) // (l * t * d))
        batch = _log_int(rng, 1, 256)
        return dict(kind=kind, n=cols * t, d=d, t=t, l=l, bits=bits,
                    log_q=log_q, batch=batch)
    if kind == "host":
        cols = _log_int(rng, 512, (1 << 29) // (l * t * d))
        return dict(kind=kind, n=cols * t, d=d, t=t, l=l, bits=bits,
                    log_q=log_q, batch=_log_int(rng, 1, 24))
    if kind == "vpir":
        d = rng.choice([1024, 2048, 4096])
        return dict(kind=kind, n=d * _log_int(rng, 1, 16), d=d, t=1,
                    l=_log_int(rng, 1, 8), bits=bits, log_q=log_q,
                    batch=_log_int(rng, 1, 24), local=rng.random() < 0.5)
    if kind == "pack":
        d = rng.choice([2048, 4096])
        return dict(kind=kind, n=_log_int(rng, 1024, 8192), d=d, t=1, l=1,
                    bits=bits, log_q=log_q, batch=_log_int(rng, 8, 256))
    if kind == "client":
        return dict(kind=kind, n=_log_int(rng, 512, 65536) * t, d=d, t=t,
                    l=l, bits=bits, log_q=log_q, batch=_log_int(rng, 1, 96))
    if kind == "interp":
        t = rng.choice([2, 4, 8])
        d = rng.choice([2048, 4096])
        return dict(kind=kind, n=_log_int(rng, 512, (1 << 29) // (t * d * l))
                    * t, d=d, t=t, l=l, value_bits=rng.choice([8, 16, 16]))
    if kind == "hint":
        cols = d * _log_int(rng, 1, 16)
        return dict(kind=kind, n=cols * t, d=d, t=t, l=1, bits=bits)
    return dict(kind="material", d=rng.choice([1024, 2048]),
                slices=_log_int(rng, 1, 8), bits=bits, log_q=log_q)


# --------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------
def _params(c):
    return synthetic.make_params(d=c["d"], n=c["n"], t=c["t"], l=c["l"],
                                 coeff_bits=c["bits"], log_q=c["log_q"])


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _words(g, shape, bits, log_q):
    """Uniform words mod 2^log_q, as int32 / int64 tensors."""
    lo = torch.randint(0, 1 << 32, shape, generator=g, device="cuda")
    if bits == 32:
        return lo.to(torch.int32)
    hi = torch.randint(0, 1 << (log_q - 32), shape, generator=g, device="cuda")
    return (hi << 32) | lo


def _u16(g, rows, cols):
    """Database words uniform in [0, 65535), as int16."""
    out = torch.empty((rows, cols), dtype=torch.int16, device="cuda")
    step = max(1, (1 << 28) // max(1, cols))
    for i in range(0, rows, step):
        m = min(step, rows - i)
        out[i:i + m] = torch.randint(0, U16_MAX, (m, cols), generator=g,
                                     device="cuda", dtype=torch.int32)
    return out


def _host(t, dtype):
    return t.cpu().numpy().view(dtype)


def _server(c, g):
    """A server over uniform material, with the pack entries and digits
    within the bounds that preprocessing gives."""
    p = _params(c)
    d, t, l, k = c["d"], c["t"], c["l"], p.pack_gadget.num_digits
    rows, cols = l * t * d, c["n"] // t
    if c["bits"] == 64:  # condensed rows of 32 records
        cols = (cols + 31) // 32 * 32
    cdt = p.coeff_dtype
    bound = int(4 * math.sqrt(d) * (1 << p.pack_gadget.log_digit))
    db = _host(_u16(g, rows, cols), np.uint16)
    pack = _host(torch.randint(-bound + 1, bound, (rows, k * d), generator=g,
                               device="cuda", dtype=torch.int32), np.int32)
    half = 1 << (p.pack_gadget.log_digit - 1)
    th = torch.randint(-half, half, (l * t * k, d), generator=g, device="cuda")
    a_tilde = _host(_words(g, (l * t, d), c["bits"], c["log_q"]), cdt)
    sda = None
    if t > 1:
        sda = _host(_words(g, (2 * p.eval_gadget.num_digits, d), c["bits"],
                           c["log_q"]), cdt)
    srv = pir.PirServer.CreateCombined(
        p, db, pack, a_tilde, th.cpu().numpy().astype(cdt), sda)
    return p, srv


def _requests(c, p, g):
    b, d = c["batch"], c["d"]
    ne = 2 * p.eval_gadget.num_digits if c["t"] > 1 else 0
    return (_words(g, (b, c["n"] // c["t"]), c["bits"], c["log_q"]),
            _words(g, (b, ne, d), c["bits"], c["log_q"]),
            _words(g, (b, 2 * p.pack_gadget.num_digits, d), c["bits"],
                   c["log_q"]))


def _word_type(c):
    return torch.int32 if c["bits"] == 32 else torch.int64


def prepare(case, seed):
    c, g = dict(case), _gen(seed)
    s = {"c": c, "kind": c["kind"]}
    return {"answer": _prepare_answer, "host": _prepare_host,
            "vpir": _prepare_vpir, "pack": _prepare_pack,
            "client": _prepare_client, "interp": _prepare_interp,
            "hint": _prepare_hint, "material": _prepare_material}[c["kind"]](
                c, g, s)


def _prepare_answer(c, g, s):
    p, srv = _server(c, g)
    fd, sd, pk = _requests(c, p, g)
    out = torch.empty((c["batch"], c["l"], 2, c["d"]), dtype=_word_type(c),
                      device="cuda")
    # A serving program tunes the tensor engine once per server for its
    # batch size.
    if c["batch"] > 4 and c["l"] * c["t"] * c["d"] % 256 == 0:
        try:
            srv.autotune(c["batch"])
        except pir.InspireError as e:
            if e.code != pir.FAILED_PRECONDITION:
                raise
    s.update(p=p, srv=srv, fd=fd, sd=sd, pk=pk, out=out)
    return s


def _prepare_host(c, g, s):
    p, srv = _server(c, g)
    fd, sd, pk = (_host(x, p.coeff_dtype) for x in _requests(c, p, g))
    s.update(p=p, srv=srv, fd=fd, sd=sd, pk=pk)
    return s


def _prepare_vpir(c, g, s):
    p, srv = _server(c, g)
    fd, _, pk = (_host(x, p.coeff_dtype) for x in _requests(c, p, g))
    if c["local"]:
        pk = np.ascontiguousarray(pk[:, :p.pack_gadget.num_digits])
    s.update(p=p, srv=pir.VpirServer(srv, c["local"]), fd=fd, pk=pk)
    return s


def _prepare_pack(c, g, s):
    # The external product belongs to the eval gadget, which a server with
    # t = 1 carries in its parameters too.
    p, srv = _server(c, g)
    b, d, ne = c["batch"], c["d"], p.eval_gadget.num_digits
    fd, _, pk = _requests(c, p, g)
    s.update(p=p, srv=srv, fd=fd, pk=pk,
             rgsw=_words(g, (b, 2 * ne, 2, d), c["bits"], c["log_q"]),
             packed=torch.empty((b, c["l"] * c["t"], 2, d),
                                dtype=_word_type(c), device="cuda"),
             out=torch.empty((b, 2, d), dtype=_word_type(c), device="cuda"))
    return s


def _prepare_client(c, g, s):
    p = _params(c)
    b, d = c["batch"], c["d"]
    k2, ne2 = 2 * p.pack_gadget.num_digits, 2 * p.eval_gadget.num_digits
    ne2 = ne2 if c["t"] > 1 else 0
    wt, cols = _word_type(c), c["n"] // c["t"]
    rows = p.NumFirstDimSamples() + ne2 + k2
    q = {"q1": p.rlwe.LogModulus1AfterSwitch(),
         "q2": p.rlwe.LogModulus2AfterSwitch()}
    resp = _words(g, (b, c["l"], 2, d), c["bits"], c["log_q"])
    resp[:, :, 0] &= (1 << q["q1"]) - 1
    resp[:, :, 1] &= (1 << q["q2"]) - 1
    s.update(
        prm=pir.c_params(p), rows=rows, resp=resp,
        keys=torch.randint(-1, 2, (b, d), generator=g, device="cuda",
                           dtype=torch.int8),
        a=_words(g, (rows, d), c["bits"], c["log_q"]),
        idx=torch.randint(0, c["n"], (b,), generator=g, device="cuda"),
        seed=int(torch.randint(0, 1 << 62, (1,), generator=g, device="cuda")),
        fd=torch.empty((b, cols), dtype=wt, device="cuda"),
        sd=torch.empty((b, ne2, d), dtype=wt, device="cuda"),
        pk=torch.empty((b, k2, d), dtype=wt, device="cuda"),
        plain=torch.empty((b, c["l"] * d), dtype=wt, device="cuda"))
    return s


def _prepare_interp(c, g, s):
    d, t, l, n = c["d"], c["t"], c["l"], c["n"]
    if c["value_bits"] == 16:
        raw, dt = _u16(g, n, l * d), torch.int16
    else:
        raw = torch.randint(0, 251, (n, l * d), generator=g, device="cuda",
                            dtype=torch.uint8)
        dt = torch.uint8
    s.update(raw=raw, modulus=U16_MAX if c["value_bits"] == 16 else 251,
             out=torch.empty((l * t * d, n // t), dtype=dt, device="cuda"))
    return s


def _prepare_hint(c, g, s):
    d, rows, cols = c["d"], c["t"] * c["d"], c["n"] // c["t"]
    s.update(db=_u16(g, rows, cols), rows=rows, cols=cols, n=cols // d,
             a=_words(g, (cols // d, d), c["bits"],
                      32 if c["bits"] == 32 else 56),
             out=torch.empty((rows, d), dtype=_word_type(c), device="cuda"))
    return s


def _prepare_material(c, g, s):
    d, sl, k, wt = c["d"], c["slices"], 2, _word_type(c)
    s.update(hint=_words(g, (sl * d, d), c["bits"], c["log_q"]),
             pa=_words(g, (2 * k, d), c["bits"], c["log_q"]), k=k,
             a_tilde=torch.empty((sl, d), dtype=wt, device="cuda"),
             matrix=torch.empty((sl * d, k * d), dtype=torch.int32,
                                device="cuda"),
             t_h=torch.empty((sl, k, d), dtype=wt, device="cuda"))
    return s


# --------------------------------------------------------------------------
# One pass
# --------------------------------------------------------------------------
def _stream():
    return torch.cuda.current_stream().cuda_stream


def _call(fn, *args):
    """A C ABI call; raises on a non-zero status, as the Python API does."""
    err = ctypes.create_string_buffer(1024)
    rc = fn(*args, err, len(err))
    if rc != 0:
        raise pir.InspireError(rc, err.value.decode(errors="replace"))


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def run(s):
    c, lib = s["c"], _lib.load()
    kind, b = s["kind"], c.get("batch", 0)
    if kind == "answer":
        s["srv"].process_device(
            b, s["fd"].data_ptr(), s["fd"].shape[1], s["sd"].data_ptr(),
            s["sd"].shape[1], s["pk"].data_ptr(), s["pk"].shape[1],
            s["out"].data_ptr(), pir.ENGINE_AUTO, _stream())
        return s["out"]
    if kind == "host":
        out = s["srv"].process_arrays(s["fd"], s["sd"], s["pk"],
                                      pir.ENGINE_AUTO)
        return out.view(np.int32 if c["bits"] == 32 else np.int64)
    if kind == "vpir":
        out = s["srv"].process_arrays(s["fd"], s["pk"], pir.ENGINE_AUTO)
        return out.view(np.int32 if c["bits"] == 32 else np.int64)
    if kind == "pack":
        st = _stream()
        s["srv"].pack_device(b, s["fd"].data_ptr(), s["fd"].shape[1],
                             s["pk"].data_ptr(), s["pk"].shape[1],
                             s["packed"].data_ptr(), pir.ENGINE_AUTO, st)
        s["srv"].external_product_device(b, s["packed"].data_ptr(),
                                         s["rgsw"].data_ptr(),
                                         s["out"].data_ptr(), st)
        return s["packed"], s["out"]
    if kind == "client":
        st = ctypes.c_void_p(_stream())
        _call(lib.inspire_client_create_requests, ctypes.byref(s["prm"]),
              _p(s["keys"]), _p(s["a"]), s["rows"], _p(s["idx"]), b,
              s["seed"], 40, _p(s["fd"]), _p(s["sd"]), _p(s["pk"]), 1, st)
        _call(lib.inspire_client_process_responses, ctypes.byref(s["prm"]),
              _p(s["keys"]), _p(s["resp"]), b, _p(s["plain"]), 1, st)
        return s["fd"], s["sd"], s["pk"], s["plain"]
    if kind == "interp":
        _call(lib.inspire_interpolate_db, c["value_bits"], _p(s["raw"]),
              s["raw"].numel(), c["n"], c["d"], c["t"], c["l"], s["modulus"],
              _p(s["out"]), s["out"].shape[1], 1, ctypes.c_void_p(_stream()))
        return s["out"]
    if kind == "hint":
        _call(lib.inspire_compute_hint_matrix, 1, c["bits"], _p(s["db"]),
              s["rows"], s["cols"], _p(s["a"]), s["n"], c["d"], _p(s["out"]),
              1, ctypes.c_void_p(_stream()))
        return s["out"]
    _call(lib.inspire_preprocess_matrix_pack, c["bits"],
          pir.KINDS[np.dtype(np.int32)], c["log_q"], 19, s["k"], c["d"],
          c["slices"], _p(s["hint"]), c["d"], _p(s["pa"]), 2 * s["k"],
          _p(s["a_tilde"]), _p(s["matrix"]), _p(s["t_h"]), 1,
          ctypes.c_void_p(_stream()))
    return s["a_tilde"], s["matrix"], s["t_h"]


# --------------------------------------------------------------------------
# What a pass cannot do without
# --------------------------------------------------------------------------
def _ntt(d):
    """Operations of one length-d transform (d / 2 log d butterflies)."""
    return 3 * d * int(math.log2(d)) // 2


def work(case):
    """Inputs read once, outputs written once; 2 operations per multiply-add
    of a matrix product, the butterflies of a polynomial product."""
    c = dict(case)
    w, d, kind = c.get("bits", 32) // 8, c["d"], c["kind"]
    if kind == "interp":
        n = c["n"] * c["l"] * d
        return {"bytes": 2 * n * c["value_bits"] // 8,
                "flops": 2 * n * max(1, int(math.log2(c["t"])))}
    if kind == "hint":
        rows, cols = c["t"] * d, c["n"] // c["t"]
        return {"bytes": 2 * rows * cols + (rows + cols // d) * d * w,
                "flops": rows * (cols // d + 1) * _ntt(d) + 2 * rows * cols}
    if kind == "material":
        sl = c["slices"]
        return {"bytes": sl * d * d * (w + 8),
                "flops": sl * (3 * d * d * int(math.log2(d)) + 3 * d * _ntt(d))}
    p = _params(c)
    b, l, t, k = c["batch"], c["l"], c["t"], p.pack_gadget.num_digits
    ne = 2 * p.eval_gadget.num_digits if t > 1 else 0
    rows, cols = l * t * d, c["n"] // t
    request = (cols + (ne + 2 * k) * d) * w
    polys = b * l * (t * (k + 1) + (t - 1) * (ne + 2)) * _ntt(d)
    if kind == "client":
        rows = p.NumFirstDimSamples() + ne + 2 * k
        return {"bytes": b * (request + d + 3 * l * d * w) + rows * d * w,
                "flops": b * (2 * rows + 1 + 2 * l) * _ntt(d)}
    out = b * l * 2 * d * w
    total = rows * (2 * cols + 4 * k * d) + b * request + out
    if kind == "pack":
        ng = 2 * p.eval_gadget.num_digits
        total += b * (2 * ng + 2) * d * w
        polys += b * (3 * ng + 2) * _ntt(d)
    return {"bytes": total,
            "flops": 2 * b * rows * (cols + k * d) + polys}


def exact(case, seed):
    """No floating outputs: the whole numbers are held bit for bit."""
    return None
