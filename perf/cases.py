"""The workloads that seedpack_b200's speed is stated on.

Each case is one call, or one short sequence of calls, that a program packing or unpacking a model repository makes through
the public entry points: re-quantising BF16 weights (`GPUQuant`), dequantising, coding a stored quantisation against its
regrown prediction and decoding it (`QRCodec`), the symbol-stream coder (`RansCodec`) and the BF16 base codec (`sg_r2_*` of
the C ABI, as the archive layer calls them).  Weights, importance matrices and symbols follow the laws of the benchmark
configurations: weights N(0, 0.02) with 0.1 % outliers at +-20 sigma, importance exp(N(0, 1.5^2)), residual symbols 97 %
zeros and Laplace(b = 2) otherwise.  Outputs are bytes (or the bit-exact floats of a dequantiser): nothing may differ.

Sizes: a row of a few thousand weights up to the 4096 x 12288 projection of the 9B shape for the quantisers, one short tensor
up to a window of 2 such tensors for the coders, 16 Ki to 256 Mi symbols for the stream coder.
"""
import ctypes

import numpy as np
import torch

from seedpack_b200 import _lib, residual
from seedpack_b200.gpuquant import GPUQuant
from seedpack_b200.qr import BS, GRID_TYPES, QK, QRCodec
from seedpack_b200.rans import RansCodec, normalize

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
SEED_TYPE = {"bf16": 30, "f16": 1, "f32": 0}
NEEDS_IMX = (16, 17, 19)                         # IQ2_XXS, IQ2_XS, IQ1_S refuse to run without a matrix
NO_IMX = (8, 42)                                 # Q8_0 and Q2_0 take none
TYPES = sorted(BS)                               # the 20 types that archives hold: Q4_0 .. Q8_0, K, IQ, Q2_0
BLOCK_LEN, NTAB = 32, 294                        # symbol stream: symbols per table id, context tables
R2_CTX, R2_PB, R2_SEG = 656, 15, 16384           # base codec: tables per role, probability bits, weights per segment


def listed():
    return [
        # the smallest call: a few rows of a matrix, where host work and launches are what counts
        dict(name="quantize-q8_0-small", op="quantize", type=8, imx=False, dtype="bf16", tensors=1, rows=16, cols=1024),
        # one layer's matrices of the 0.6B shape in one launch with the type that most repositories carry
        dict(name="quantize-q4_k-imx", op="quantize", type=12, imx=True, dtype="bf16", tensors=4, rows=1024, cols=3072),
        # a whole projection of the 9B shape without an importance matrix
        dict(name="quantize-q6_k-large", op="quantize", type=14, imx=False, dtype="bf16", tensors=1, rows=4096, cols=12288),
        # a lattice type: a search through the grid's neighbours for every group of weights
        dict(name="quantize-iq2_xs-imx", op="quantize", type=17, imx=True, dtype="bf16", tensors=1, rows=4096, cols=4096),
        # an odd number of rows that do not fill whole slabs, from an F16 model, with the older importance arithmetic
        dict(name="quantize-q5_1-imx-ragged", op="quantize", type=7, imx=True, dtype="f16", tensors=3, rows=1001, cols=2080),
        # a sibling quantisation turned back into weights
        dict(name="dequantize-q4_k", op="dequantize", type=12, rows=4096, cols=4096),
        # the residual symbol coder, there and back
        dict(name="symbols-round-trip", op="symbols", nsym=1 << 27, zeros=0.97),
        # a stored file against its prediction: compare, model, code (pack)
        dict(name="residual-encode-q4_k", op="encode", type=12, dtype="bf16", tensors=2, rows=4096, cols=4096),
        # the same back from the archive (unpack), and the lattice form of it
        dict(name="residual-decode-q4_k", op="decode", type=12, dtype="bf16", tensors=2, rows=4096, cols=4096),
        dict(name="residual-decode-iq3_s", op="decode", type=21, dtype="bf16", tensors=1, rows=1024, cols=3072),
        # the BF16 base file: statistics, duplicate-row hashes, histogram, tables, code; and its decoder
        dict(name="base-encode", op="base-encode", tensors=2, rows=4096, cols=12288),
        dict(name="base-decode", op="base-decode", tensors=2, rows=4096, cols=12288),
    ]


def _spread(rng, lo, hi):
    """a whole number between lo and hi, even over its logarithm"""
    return int(round(lo * (hi / lo) ** rng.random()))


def _matrix(rng, unit, most, least=1):
    """rows and columns of one tensor: columns whole blocks of `unit` up to 17408, `least` .. `most` weights in all"""
    total = _spread(rng, max(least, 4096), most)
    cols = _spread(rng, max(1, 256 // unit), 17408 // unit) * unit
    cols = min(cols, max(unit, total // unit * unit))
    return max(1, total // cols), cols


def draw(rng):
    op = rng.choices(("quantize", "dequantize", "symbols", "encode", "decode", "base-encode", "base-decode"), (40, 8, 10, 12, 12, 9, 9))[0]
    dtype = rng.choices(("bf16", "f16", "f32"), (8, 1, 1))[0]
    t = rng.choice(TYPES)
    if op == "quantize":
        tensors = rng.choice((1, 1, 1, 2, 3, 5, 8, 20))
        rows, cols = _matrix(rng, QK[t], 4096 * 12288 // tensors)
        imx = t in NEEDS_IMX or (t not in NO_IMX and rng.random() < 0.6)
        return dict(op=op, type=t, imx=imx, dtype=dtype, tensors=tensors, rows=rows, cols=cols)
    if op == "dequantize":
        rows, cols = _matrix(rng, QK[t], 4096 * 12288)
        return dict(op=op, type=t, rows=rows, cols=cols)
    if op == "symbols":
        return dict(op=op, nsym=_spread(rng, 1 << 14, 1 << 27) // BLOCK_LEN * BLOCK_LEN, zeros=round(rng.uniform(0.9, 0.99), 3))
    tensors = rng.choice((1, 2, 3, 4))
    if op in ("encode", "decode"):
        # a lattice type's ranking of all its points costs some ten times a scalar code's model
        rows, cols = _matrix(rng, QK[t], (1 << 22 if t in GRID_TYPES else 1 << 25) // tensors, 1 << 15)
        return dict(op=op, type=t, dtype=dtype, tensors=tensors, rows=rows, cols=cols)
    rows, cols = _matrix(rng, 32, 2 * 4096 * 12288 // tensors, 1 << 16)
    return dict(op=op, tensors=tensors, rows=rows, cols=cols)


# ---- inputs -------------------------------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _weights(n, g, dtype):
    x = torch.randn(n, generator=g, device="cuda") * 0.02
    u = torch.rand(n, generator=g, device="cuda")
    x = torch.where(u < 0.0005, -0.4, torch.where(u > 0.9995, 0.4, x))
    return x.to(torch.bfloat16).to(DTYPES[dtype])


def _importance(n, g, spread=1.5):
    return torch.exp(torch.randn(n, generator=g, device="cuda") * spread)


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _call(name, *args):
    _lib.check(getattr(_lib.lib(), name)(torch.cuda.current_device(), _stream(), *args), name)


def _window(case, seed):
    """tensors back to back as in a window of the base file, one importance vector per tensor"""
    g = _gen(seed)
    k, rows, cols = case["tensors"], case["rows"], case["cols"]
    buf = _weights(k * rows * cols, g, case["dtype"])
    return g, buf, list(buf.view(k, -1).unbind(0)), [_importance(cols, g) for _ in range(k)]


def prepare(case, seed):
    return globals()["_prepare_" + case["op"].replace("-", "_")](case, seed)


def _prepare_quantize(case, seed):
    _, _, xs, imx = _window(case, seed)
    return dict(case=case, gq=GPUQuant(), srcs=[(x, case["cols"]) for x in xs], imx=imx if case["imx"] else [None] * len(xs))


def _prepare_dequantize(case, seed):
    t = case["type"]
    _, _, xs, imx = _window(dict(case, tensors=1, dtype="bf16"), seed)
    gq = GPUQuant()
    return dict(case=case, gq=gq, y=gq.quantize_tensors(t, [(xs[0], case["cols"])], imx if t not in NO_IMX else [None], device=True)[0])


def _prepare_symbols(case, seed):
    """blocks of 32 symbols with an alphabet of 4 / 5 / 6 / 8 bits and a context table each"""
    g = _gen(seed)
    n = case["nsym"]
    kind = torch.randint(0, 4, (n // BLOCK_LEN,), generator=g, device="cuda")
    tab = (kind * 73 + torch.randint(0, 73, kind.shape, generator=g, device="cuda")).to(torch.int16)
    mask = torch.tensor([15, 31, 63, 255], dtype=torch.uint8, device="cuda")[kind]
    sym = torch.empty(n, dtype=torch.uint8, device="cuda")
    for a in range(0, n, 1 << 25):
        m = min(1 << 25, n - a)
        mag = torch.floor(-2.0 * torch.log(torch.rand(m, generator=g, device="cuda").clamp_min(1e-12))).to(torch.int16)
        v = torch.where(torch.rand(m, generator=g, device="cuda") < 0.5, mag, -mag)
        v = torch.where(torch.rand(m, generator=g, device="cuda") < case["zeros"], 0, v) & 255
        sym[a:a + m] = v.to(torch.uint8) & mask[a // BLOCK_LEN:(a + m) // BLOCK_LEN].repeat_interleave(BLOCK_LEN)
    return dict(case=case, codec=RansCodec(), sym=sym, tab=tab, archive=torch.zeros(n + 65536, dtype=torch.uint8, device="cuda"))


def _stored_and_predicted(case, seed):
    """what pack holds of one batch: stored blocks (made with a slightly different importance matrix; one byte flipped in
    0.5 % of the blocks), the prediction regrown from the base, the base's bytes and the importance vectors"""
    t, k, cols = case["type"], case["tensors"], case["cols"]
    g, buf, xs, imx = _window(case, seed)
    gq = GPUQuant()
    srcs = [(x, cols) for x in xs]
    takes = t not in NO_IMX
    pred = gq.quantize_tensors(t, srcs, imx if takes else [None] * k, device=True)
    other = [w * _importance(cols, g, 0.3) for w in imx]
    files = [f.clone() for f in gq.quantize_tensors(t, srcs, other if takes else [None] * k, device=True)]
    for f in files:
        nb = f.numel() // BS[t]
        hit = torch.nonzero(torch.rand(nb, generator=g, device="cuda") < 0.005).reshape(-1)
        at = hit * BS[t] + torch.randint(0, BS[t], hit.shape, generator=g, device="cuda")
        f[at] ^= torch.randint(1, 256, hit.shape, generator=g, device="cuda").to(torch.uint8)
    step = case["rows"] * cols * buf.element_size()
    grid = t in GRID_TYPES
    enc = [(files[i], pred[i], i * step, SEED_TYPE[case["dtype"]], cols, i * cols if grid else -1) for i in range(k)]
    return dict(case=case, codec=QRCodec(), enc=enc, seed=buf.view(torch.uint8), imx=torch.cat(imx) if grid else None,
                archive=np.zeros(sum(f.numel() for f in files) + (1 << 18), np.uint8))


def _prepare_encode(case, seed):
    return _stored_and_predicted(case, seed)


def _prepare_decode(case, seed):
    s = _stored_and_predicted(case, seed)
    s["coded"] = s["codec"].encode(case["type"], s["enc"], s["seed"], s["imx"])
    s["dec"] = [it[1:] for it in s.pop("enc")]
    return s


def _base_layout(case, seed):
    """one group of the base file: tensors of one role, and the records that the coder's launches share"""
    k, rows, cols = case["tensors"], case["rows"], case["cols"]
    n = rows * cols
    w = _window(dict(case, dtype="bf16"), seed)[1]
    per = -(-n // R2_SEG)
    tb = np.zeros(k, np.dtype([("doff", "<i8"), ("rowlen", "<i4"), ("rowbase", "<i4"), ("colbase", "<i4"), ("tab", "<i4"), ("rmap", "<i4"),
                               ("pad", "<i4")]))
    sg = np.zeros(k * per, np.dtype([("t", "<i4"), ("n", "<i4"), ("i0", "<i8")]))
    for i in range(k):
        tb[i] = (i * n * 2, cols, i * rows, i * cols, 0, -1, 0)
        i0 = np.arange(per, dtype=np.int64) * R2_SEG
        part = sg[i * per:(i + 1) * per]
        part["t"], part["i0"], part["n"] = i, i0, np.minimum(R2_SEG, n - i0)
    scratch = _lib.lib().sg_r2_stats_scratch_bytes(rows, cols)
    return dict(case=case, w=w, tb=torch.from_numpy(tb.view(np.uint8)).cuda(), sg=torch.from_numpy(sg.view(np.uint8)).cuda(), nseg=len(sg),
                scratch=torch.empty(scratch, dtype=torch.uint8, device="cuda"), rowmap=torch.zeros(1, dtype=torch.int32, device="cuda"),
                archive=torch.zeros(2 * k * n + 65536, dtype=torch.uint8, device="cuda"))


def _prepare_base_encode(case, seed):
    return _base_layout(case, seed)


def _prepare_base_decode(case, seed):
    s = _base_layout(case, seed)
    out = _run_base_encode(s)
    s.pop("w")
    s.update(coded=s.pop("archive"), first=out["off"][:-1], end=out["off"][1:], freq=out["freq"], rfi=out["rfi"], cfi=out["cfi"], scl=out["scl"])
    return s


# ---- one pass -----------------------------------------------------------------------------------------------------------
# Coded bytes go to the place in the archive that the program holds for them (`archive`): their number depends on the data.
def run(state):
    return globals()["_run_" + state["case"]["op"].replace("-", "_")](state)


def _run_quantize(s):
    return s["gq"].quantize_tensors(s["case"]["type"], s["srcs"], s["imx"], device=True)


def _run_dequantize(s):
    return s["gq"].dequantize(s["case"]["type"], s["y"])


def _all_rows(ntab, freq, used):
    full = np.zeros((ntab, 256), np.uint16)
    full[used] = freq
    return full


def _run_symbols(s):
    c, n = s["codec"], s["case"]["nsym"]
    r = c.encode(s["sym"], s["tab"], BLOCK_LEN, NTAB)
    back = c.decode(r["stream"], r["off"], s["tab"], BLOCK_LEN, n, r["freq"], r["used"], NTAB)
    s["archive"][:r["total"]] = r["stream"][:r["total"]]
    return s["archive"], r["off"], _all_rows(NTAB, r["freq"], r["used"]), back


def _run_encode(s):
    differ = [residual.count_diff(it[0], it[1], sync=False) for it in s["enc"]]
    coded = s["codec"].encode(s["case"]["type"], s["enc"], s["seed"], s["imx"])
    s["archive"][:len(coded)] = np.frombuffer(coded, np.uint8)
    return s["archive"], len(coded), differ


def _run_decode(s):
    return s["codec"].decode(s["case"]["type"], s["coded"], s["dec"], s["seed"], s["imx"])


def _tables(full, lut):
    enc = torch.empty(R2_CTX * 256 * 2, dtype=torch.int32, device="cuda")
    compact = torch.empty(R2_CTX * 1280, dtype=torch.uint8, device="cuda") if lut else None
    f = torch.from_numpy(full.view(np.int16)).cuda()
    _call("sg_rans_tables", _ptr(f), R2_CTX, R2_PB, _ptr(enc), _ptr(compact))
    return enc, compact


def _run_base_encode(s):
    """a group of the base file as the archive layer codes it (statistics and row hashes per tensor, one histogram, tables
    normalised on the host, one coder launch, the segments gathered)"""
    k, rows, cols, nseg, w = s["case"]["tensors"], s["case"]["rows"], s["case"]["cols"], s["nseg"], s["w"]
    rfi = torch.empty(k * rows, dtype=torch.int16, device="cuda")
    cfi = torch.empty(k * cols, dtype=torch.int16, device="cuda")
    scl = torch.empty(k * cols, dtype=torch.int8, device="cuda")
    hashes = torch.empty(k * rows, dtype=torch.int64, device="cuda")
    for i in range(k):
        x = w[i * rows * cols:(i + 1) * rows * cols]
        _call("sg_r2_stats", _ptr(x), rows, cols, _ptr(rfi[i * rows:]), _ptr(cfi[i * cols:]), _ptr(scl[i * cols:]), _ptr(s["scratch"]),
              s["scratch"].numel())
        _call("sg_row_hash", _ptr(x), rows, cols, _ptr(hashes[i * rows:]))
    side = (_ptr(rfi), _ptr(cfi), _ptr(scl), _ptr(s["rowmap"]))
    counts = torch.zeros(R2_CTX * 256, dtype=torch.int32, device="cuda")
    _call("sg_r2_hist", _ptr(w), _ptr(s["tb"]), _ptr(s["sg"]), nseg, *side, _ptr(counts))
    freq, used = normalize(counts.cpu().numpy().reshape(R2_CTX, 256), 1 << R2_PB)
    full = _all_rows(R2_CTX, freq, used)
    enc, _ = _tables(full, False)
    cap = R2_SEG * 2 + 1024
    slots = torch.empty(nseg * cap, dtype=torch.uint8, device="cuda")
    lens = torch.empty(nseg, dtype=torch.int32, device="cuda")
    _call("sg_r2_encode", _ptr(w), _ptr(s["tb"]), _ptr(s["sg"]), nseg, *side, _ptr(enc), _ptr(slots), cap, _ptr(lens))
    total = int(lens.cpu().numpy().astype(np.int64).sum())
    off = torch.empty(nseg + 1, dtype=torch.int64, device="cuda")
    _call("sg_scan_gather", _ptr(slots), cap, _ptr(lens), nseg, _ptr(s["archive"]), total, _ptr(off))
    return dict(stream=s["archive"], off=off, freq=full, rfi=rfi, cfi=cfi, scl=scl, hashes=hashes)


def _run_base_decode(s):
    enc, compact = _tables(s["freq"], True)
    w = torch.empty(s["case"]["tensors"] * s["case"]["rows"] * s["case"]["cols"], dtype=torch.int16, device="cuda")
    _call("sg_r2_decode", _ptr(s["coded"]), _ptr(s["first"]), _ptr(s["end"]), _ptr(w), _ptr(s["tb"]), _ptr(s["sg"]), s["nseg"], _ptr(s["rfi"]),
          _ptr(s["cfi"]), _ptr(s["scl"]), _ptr(s["rowmap"]), _ptr(enc), _ptr(compact))
    return w


# ---- what a pass cannot do without ----------------------------------------------------------------------------------------
def work(case):
    """bytes that have to be read and written once.  No operation count: the quantisers are scalar searches and the coders
    dependent integer chains, nothing here is a contraction that a peak in FLOP/s would bound"""
    op = case["op"]
    if op == "symbols":
        n = case["nsym"]
        coded = n * (1 - case["zeros"]) * 5 / 8 + n * 0.02
        return {"bytes": 2 * (n + n // BLOCK_LEN * 2) + 2 * coded, "flops": 0}
    n = case.get("tensors", 1) * case["rows"] * case["cols"]
    if op in ("base-encode", "base-decode"):
        return {"bytes": 2 * n + 1.4 * n, "flops": 0}
    t = case["type"]
    q = n // QK[t] * BS[t]
    if op == "dequantize":
        return {"bytes": q + 4 * n, "flops": 0}
    w = n * torch.empty(0, dtype=DTYPES[case["dtype"]]).element_size()
    if op == "quantize":
        return {"bytes": w + q + (4 * case["tensors"] * case["cols"] if case["imx"] else 0), "flops": 0}
    return {"bytes": 2 * q + w + 0.1 * q, "flops": 0}


def tolerance(case):
    return "exact"
