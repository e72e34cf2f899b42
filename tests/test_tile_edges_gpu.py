"""Kernels at the sizes where their tiles, batches and remainders end."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", [2, 3, 6, 7, 8, 10, 11, 12, 13, 14, 16, 17, 18, 19, 20, 21, 22, 23, 29, 42])
def test_dequantize_tiles(t):
    """a tensor dequantised in tiles equals its blocks dequantised one by one, whatever the alignment of the bytes: one block, a
    tile less one block, a tile, one block more (exact: the same operations per weight)"""
    import torch
    from seedpack_b200.gpuquant import GPUQuant
    from seedpack_b200.requant import QFUN
    gq = GPUQuant()
    _, qk, bs = QFUN[t]
    tile = 4096 // qk
    y = torch.from_numpy(np.random.default_rng(t).integers(0, 256, (tile + 2) * bs, dtype=np.uint8)).cuda()
    alone = torch.cat([gq.dequantize(t, y[i * bs:(i + 1) * bs].clone()) for i in (0, tile - 1, tile)]).view(torch.int32)
    for nb in (1, tile - 1, tile, tile + 1):
        for off in (0, 2):
            buf = torch.zeros(nb * bs + 16, dtype=torch.uint8, device="cuda")
            buf[off:off + nb * bs] = y[:nb * bs]
            got = gq.dequantize(t, buf[off:off + nb * bs]).view(torch.int32)
            for k, i in enumerate((0, tile - 1, tile)):
                if i < nb:
                    assert torch.equal(got[i * qk:(i + 1) * qk], alone[k * qk:(k + 1) * qk]), (nb, off, i)


def test_dequantize_values():
    """Q8_0 and Q4_0 against the formulas in NumPy (one product per weight, exact)"""
    import torch
    from seedpack_b200.gpuquant import GPUQuant
    gq = GPUQuant()
    rng = np.random.default_rng(1)
    d = (rng.random(300).astype(np.float32) * 2 - 1).astype(np.float16)
    q8 = rng.integers(-128, 128, (300, 32)).astype(np.int8)
    y = np.concatenate([d.view(np.uint8).reshape(-1, 2), q8.view(np.uint8)], 1)
    want = q8.astype(np.float32) * d.astype(np.float32)[:, None]
    assert np.array_equal(gq.dequantize(8, torch.from_numpy(y).cuda()).cpu().numpy().reshape(-1, 32), want)
    q4 = rng.integers(0, 16, (300, 32)).astype(np.uint8)
    y = np.concatenate([d.view(np.uint8).reshape(-1, 2), q4[:, :16] | (q4[:, 16:] << 4)], 1)
    want = (q4.astype(np.float32) - 8) * d.astype(np.float32)[:, None]
    assert np.array_equal(gq.dequantize(2, torch.from_numpy(y).cuda()).cpu().numpy().reshape(-1, 32), want)


@pytest.mark.parametrize("t", [2, 3, 6, 7, 8, 10, 11, 12, 13, 14, 16, 17, 18, 19, 20, 21, 22, 23, 29, 42])
def test_dequantize_equals_the_formulas(t):
    """random blocks against the layouts and formulas in NumPy, exact (NaN where the scale is one)"""
    import torch
    from seedpack_b200.gpuquant import GPUQuant
    from seedpack_b200.requant import QFUN
    from tests.dequant_model import dequantize
    _, qk, bs = QFUN[t]
    y = np.random.default_rng(100 + t).integers(0, 256, (4096 // qk + 300) * bs, dtype=np.uint8)
    got = GPUQuant().dequantize(t, torch.from_numpy(y).cuda()).cpu().numpy()
    assert np.array_equal(got.reshape(-1, qk), dequantize(t, y, bs), equal_nan=True)


R2_SHAPES = [(1, 1, 0), (5, 37, 0), (3, 16384, 0), (64, 1000, 1), (700, 4099, 1)]


@pytest.mark.parametrize("rows,cols,spread", R2_SHAPES)
def test_base_codec_round_trip(rows, cols, spread):
    """two tensors of different roles in one launch: segments of one weight and of ragged batches, and (spread) rows over more
    octaves than the decoder stages tables for, zeros and infinities among them: the weights come back bit for bit"""
    import ctypes

    import torch
    from seedpack_b200 import _lib
    from seedpack_b200.rans import normalize
    L, dev = _lib.lib(), torch.device("cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    call = lambda name, *a: _lib.check(getattr(L, name)(torch.cuda.current_device(), st, *a), name)
    g = torch.Generator(device="cuda").manual_seed(rows * cols)
    w = torch.randn(2, rows, cols, generator=g, device=dev)
    if spread:
        w *= torch.exp2(torch.randint(-40, 40, (2, rows, 1), generator=g, device=dev).float())
        w[:, ::7, ::11] = 0
        w[1, 0, 0] = float("inf")
    w = w.to(torch.bfloat16).view(torch.int16).reshape(-1)
    n, ntab = rows * cols, 2 * 656
    tb = np.zeros(2, np.dtype([("doff", "<i8"), ("rowlen", "<i4"), ("rowbase", "<i4"), ("colbase", "<i4"), ("tab", "<i4"), ("rmap", "<i4"), ("pad", "<i4")]))
    segs = []
    for i in range(2):
        tb[i] = (2 * i * n, cols, i * rows, i * cols, i * 656, -1, 0)
        segs += [(i, min(16384, n - a), a) for a in range(0, n, 16384)]
    sg = np.array(segs, np.dtype([("t", "<i4"), ("n", "<i4"), ("i0", "<i8")]))
    tb, sg, nseg = torch.from_numpy(tb.view(np.uint8)).cuda(), torch.from_numpy(sg.view(np.uint8)).cuda(), len(sg)
    rfi, cfi = torch.empty(2 * rows, dtype=torch.int16, device=dev), torch.empty(2 * cols, dtype=torch.int16, device=dev)
    scl = torch.empty(2 * cols, dtype=torch.int8, device=dev)
    scratch = torch.empty(L.sg_r2_stats_scratch_bytes(rows, cols), dtype=torch.uint8, device=dev)
    for i in range(2):
        call("sg_r2_stats", p(w[i * n:]), rows, cols, p(rfi[i * rows:]), p(cfi[i * cols:]), p(scl[i * cols:]), p(scratch), scratch.numel())
    none = torch.zeros(1, dtype=torch.int32, device=dev)
    side = (p(rfi), p(cfi), p(scl), p(none))
    counts = torch.zeros(ntab * 256, dtype=torch.int32, device=dev)
    call("sg_r2_hist", p(w), p(tb), p(sg), nseg, *side, p(counts))
    h = counts.cpu().numpy().reshape(ntab, 256)
    assert h.sum() == 6 * n
    # the histogram against NumPy, over the side information the device made
    u = w.cpu().numpy().view(np.uint16).reshape(2, rows, cols).astype(np.int64)
    pred = rfi.cpu().numpy().reshape(2, rows, 1).astype(np.int64) + cfi.cpu().numpy().reshape(2, 1, cols)
    ex, base = (u >> 7) & 255, np.arange(2).reshape(2, 1, 1) * 656
    want = np.zeros(ntab * 256, np.int64)
    for tab, sym in ((np.clip(pred + 256, 0, 511), ex), (512 + np.clip(8 * ex - pred - 952, 0, 127), u & 127),
                     (640 + np.clip(scl.cpu().numpy().reshape(2, 1, cols).astype(np.int64), 0, 15) + 0 * ex, u >> 15)):
        want += np.bincount(((base + tab) * 256 + sym).reshape(-1), minlength=ntab * 256)
    assert np.array_equal(h.reshape(-1), want)
    freq, used = normalize(h, 1 << 15)
    full = np.zeros((ntab, 256), np.uint16)
    full[used] = freq
    f = torch.from_numpy(full.view(np.int16)).cuda()
    enc, lut = torch.empty(ntab * 512, dtype=torch.int32, device=dev), torch.empty(ntab * 1280, dtype=torch.uint8, device=dev)
    call("sg_rans_tables", p(f), ntab, 15, p(enc), p(lut))
    cap = 16384 * 4 + 1024
    slots, lens = torch.empty(nseg * cap, dtype=torch.uint8, device=dev), torch.empty(nseg, dtype=torch.int32, device=dev)
    call("sg_r2_encode", p(w), p(tb), p(sg), nseg, *side, p(enc), p(slots), cap, p(lens))
    total = int(lens.cpu().numpy().view(np.uint32).astype(np.int64).sum())
    assert 0 < total < nseg * cap
    stream, off = torch.zeros((total + 31) // 16 * 16, dtype=torch.uint8, device=dev), torch.empty(nseg + 1, dtype=torch.int64, device=dev)
    call("sg_scan_gather", p(slots), cap, p(lens), nseg, p(stream), total, p(off))
    back = torch.full_like(w, -1)
    call("sg_r2_decode", p(stream), p(off), p(off[1:]), p(back), p(tb), p(sg), nseg, *side, p(enc), p(lut))
    bits = ctypes.c_int(0)
    _lib.check(L.sg_status_fetch(torch.cuda.current_device(), st, ctypes.byref(bits)), "sg_status_fetch")
    assert bits.value == 0 and torch.equal(back, w)


@pytest.mark.parametrize("rows,cols,off", [(1, 1, 0), (33, 64, 0), (31, 72, 0), (40, 130, 0), (5, 1001, 0), (32, 256, 2), (7, 256, 1),
                                           (1, 1, 1), (2, 2, 1), (3, 63, 1), (9, 65, 7), (34, 127, 1), (4, 4033, 3), (9, 8, 4), (9, 7, 0)])
def test_row_recurrences(rows, cols, off):
    """row fingerprints and row statistics against the recurrences in Python (integers; float64 sums in order), for rows whose
    length and address are multiples of 16 bytes, and for rows that begin and end anywhere within them"""
    import ctypes

    import torch
    from seedpack_b200 import _lib
    L = _lib.lib()
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    rng = np.random.default_rng(rows * cols)
    w32 = (rng.standard_normal((rows, cols)) * 0.02).astype(np.float32)
    bits = (w32.view(np.uint32) >> 16).astype(np.uint16)
    buf = torch.zeros(off + rows * cols + 8, dtype=torch.int16, device="cuda")
    w = buf[off:off + rows * cols]
    w.copy_(torch.from_numpy(bits.view(np.int16).reshape(-1)))
    h = torch.zeros(rows, dtype=torch.int64, device="cuda")
    _lib.check(L.sg_row_hash(0, st, p(w), rows, cols, p(h)), "sg_row_hash")
    rfi, cfi = torch.zeros(rows, dtype=torch.int16, device="cuda"), torch.zeros(cols, dtype=torch.int16, device="cuda")
    scl, scratch = torch.zeros(cols, dtype=torch.int8, device="cuda"), torch.zeros(L.sg_r2_stats_scratch_bytes(rows, cols), dtype=torch.uint8, device="cuda")
    _lib.check(L.sg_r2_stats(0, st, p(w), rows, cols, p(rfi), p(cfi), p(scl), p(scratch), scratch.numel()), "sg_r2_stats")
    for r in range(rows):
        a, s = 1469598103934665603, 0.0
        for v in bits[r].tolist():
            a = ((a ^ v) * 1099511628211) & (2 ** 64 - 1)
            a ^= a >> 29
        for v in (bits[r].astype(np.uint32) << 16).view(np.float32).astype(np.float64).tolist():
            s += v * v
        assert int(h[r]) & (2 ** 64 - 1) == a
        lg = 8 * np.log2(np.sqrt(s / cols) + 1e-30)
        assert abs(int(rfi[r]) - lg) <= 0.5 + 1e-9            # round to nearest; log2 to well below 1e-9


@pytest.mark.parametrize("t", [16, 17, 18, 19, 21, 22, 29])
def test_lattice_points_at_equal_distances(t):
    """residual batches of the lattice types come back bit for bit where many of a group's lattice points lie equally far from the
    seed: weights of few magnitudes, zeros among them, columns without importance.  Every rank occurs, the ones that
    the decoder ranks ahead and the ones that it looks up."""
    import torch
    from seedpack_b200.gpuquant import GPUQuant
    from seedpack_b200.qr import QRCodec
    rows, cols = 96, 3072
    g = torch.Generator(device="cuda").manual_seed(t)
    pick = lambda n, values, p: torch.tensor(values, device="cuda")[torch.multinomial(torch.tensor(p), n, replacement=True, generator=torch.Generator().manual_seed(t)).cuda()]
    x = pick(rows * cols, [-2.0, -1.0, 0.0, 1.0, 2.0], [0.1, 0.35, 0.1, 0.35, 0.1]) * 0.0625
    x[:cols] = 0.0625                                            # a row of one value, and one of zeros
    x[cols:2 * cols] = 0
    x = x.to(torch.bfloat16)
    imx = pick(cols, [0.0, 1.0], [0.1, 0.9]).float()
    gq, codec = GPUQuant(), QRCodec()
    pred = gq.quantize_tensors(t, [(x, cols)], [imx], device=True)[0]
    noise = torch.where(torch.rand(rows * cols, generator=g, device="cuda") < 0.3, torch.randn(rows * cols, generator=g, device="cuda") * 0.05, 0)
    file = gq.quantize_tensors(t, [((x.float() + noise).to(torch.bfloat16), cols)], [torch.ones_like(imx)], device=True)[0].clone()
    seed = x.view(torch.uint8)
    _, counts = codec.hist(t, [(file, pred, 0, 30, cols, 0)], seed, imx)
    ranks = counts[214:230].sum(0)                               # the tables of the ranks; 16: a rank past the list's end
    assert (ranks[:5] > 50).all() and ranks[4:16].sum() > 100 and ranks[16] > 50, ranks[:17]
    buf = codec.encode(t, [(file, pred, 0, 30, cols, 0)], seed, imx)
    assert torch.equal(codec.decode(t, buf, [(pred, 0, 30, cols, 0)], seed, imx), file)


def _quantised_pair(t, n, cols, seed, importance=None):
    """n weights, and their blocks of type t as a prediction and as a file made from slightly other weights"""
    import torch
    from seedpack_b200.gpuquant import GPUQuant
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = (torch.randn(n, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    y = torch.where(torch.rand(n, generator=g, device="cuda") < 0.1, x + torch.randn(n, generator=g, device="cuda") * 0.01, x.float()).to(torch.bfloat16)
    pred, file = (GPUQuant().quantize_tensors(t, [(v, cols)], [importance], device=True)[0].clone() for v in (x, y))
    return x, pred, file


@pytest.mark.parametrize("t", [2, 3, 6, 7, 8, 10, 11, 12, 13, 14, 20, 23, 42])
def test_residual_decoder_with_many_segments(t):
    """more segments than five CTAs a SM take, of one and two blocks (a tensor each), the last CTA partly filled"""
    import torch
    from seedpack_b200.qr import BS, QK, QRCodec
    nseg, qk, bs = 148 * 5 * 16 + 5, QK[t], BS[t]
    nb = nseg + nseg // 3
    x, pred, file = _quantised_pair(t, nb * qk, qk, t)
    items, b = [], 0
    for i in range(nseg):
        k = 2 if i < nseg // 3 else 1
        items.append((file[b * bs:(b + k) * bs], pred[b * bs:(b + k) * bs], 2 * b * qk, 30, qk))
        b += k
    codec, seed = QRCodec(), x.view(torch.uint8)
    assert 0.05 < (file.view(nb, bs) != pred.view(nb, bs)).any(1).float().mean() <= 1
    buf = codec.encode(t, items, seed)
    assert torch.equal(codec.decode(t, buf, [it[1:] for it in items], seed), file)


@pytest.mark.parametrize("t", [16, 17, 18, 19, 21, 22, 29])
def test_lattice_decoder_with_many_segments(t):
    """more segments than the kernel of eight warps is used for, of one to three blocks (a tensor each); blocks that equal their
    prediction and blocks that do not follow one another in every order"""
    import torch
    from seedpack_b200.qr import BS, QRCodec
    nseg, bs = 148 * 4 + 1, BS[t]
    sizes = [1 + i % 3 for i in range(nseg)]
    nb = sum(sizes)
    imx = torch.linspace(0.5, 2.0, 256, device="cuda")
    x, pred, file = _quantised_pair(t, nb * 256, 256, t, imx)
    keep = torch.rand(nb, generator=torch.Generator(device="cuda").manual_seed(t), device="cuda") < 0.5
    file = torch.where(keep[:, None], pred.view(nb, bs), file.view(nb, bs)).reshape(-1)
    items, b = [], 0
    for k in sizes:
        items.append((file[b * bs:(b + k) * bs], pred[b * bs:(b + k) * bs], 2 * b * 256, 30, 256, 0))
        b += k
    codec, seed = QRCodec(), x.view(torch.uint8)
    buf = codec.encode(t, items, seed, imx)
    assert torch.equal(codec.decode(t, buf, [it[1:] for it in items], seed, imx), file)
    one = [(file, pred, 0, 30, 256, 0)]                          # the same blocks in few segments
    buf = codec.encode(t, one, seed, imx)
    assert torch.equal(codec.decode(t, buf, [it[1:] for it in one], seed, imx), file)


# how the base decoder cuts its segments: one wave of CTAs with several chains a warp, two waves, runs of two roles, runs too short to
# be decoded with the role's tables staged (four waves of them; more runs than the kernel lists), a table the stage has no room for,
# rows over more octaves than it has room for
BASE_CUTS = {
    "one role": (12000, lambda i: 0, None, 24), "two waves": (15000, lambda i: 0, None, 24), "runs": (9001, lambda i: i // 700 % 3, None, 24),
    "short runs": (500, lambda i: i % 2, None, 24), "many runs": (1100, lambda i: i % 2, None, 24),
    "symbol past 127": (600, lambda i: i // 300, 200, 24), "many octaves": (5000, lambda i: i // 1000, None, 200),
}


@pytest.mark.parametrize("name", BASE_CUTS)
def test_base_decoder_cuts(name):
    """many segments of 1 to 100 weights, rows over several octaves and some zeros: the weights come back bit for bit"""
    import ctypes

    import torch
    from seedpack_b200 import _lib
    from seedpack_b200.rans import normalize
    nseg, role, extra, spread = BASE_CUTS[name]
    L, dev = _lib.lib(), torch.device("cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    call = lambda fn, *a: _lib.check(getattr(L, fn)(0, st, *a), fn)
    rng = np.random.default_rng(len(name))
    ns = rng.integers(1, 101, nseg)
    roles = np.array([role(i) for i in range(nseg)])
    starts = np.flatnonzero(np.r_[True, roles[1:] != roles[:-1]])                # a tensor per run of one role, of 37 columns
    ends = np.r_[starts[1:], nseg]
    cols, sizes = 37, np.array([int(ns[a:b].sum()) for a, b in zip(starts, ends)])
    rows = -(-sizes // cols)
    rowbase = np.r_[0, np.cumsum(rows)]
    at = int(rowbase[-1]) * cols
    tb = np.zeros(len(sizes), np.dtype([("doff", "<i8"), ("rowlen", "<i4"), ("rowbase", "<i4"), ("colbase", "<i4"), ("tab", "<i4"), ("rmap", "<i4"), ("pad", "<i4")]))
    segs = []
    for t, (a, b) in enumerate(zip(starts, ends)):
        tb[t] = (2 * rowbase[t] * cols, cols, rowbase[t], t * cols, roles[a] * 656, -1, 0)
        segs += list(zip([t] * (b - a), ns[a:b].tolist(), (np.cumsum(ns[a:b]) - ns[a:b]).tolist()))
    sg = np.array(segs, np.dtype([("t", "<i4"), ("n", "<i4"), ("i0", "<i8")]))
    tb, sg = torch.from_numpy(tb.view(np.uint8)).cuda(), torch.from_numpy(sg.view(np.uint8)).cuda()
    g = torch.Generator(device="cuda").manual_seed(nseg)
    w = torch.randn(at, generator=g, device=dev) * torch.exp2(torch.randint(-3, 4, (at // cols, 1), generator=g, device=dev).float()).expand(-1, cols).reshape(-1)
    w = torch.where(torch.rand(at, generator=g, device=dev) < 0.01, 0, w).to(torch.bfloat16).view(torch.int16)
    # side information from the weights: whole eighths of an octave a row and a column, a class a column
    rfi = torch.randint(-spread, spread + 1, (at // cols,), generator=g, device=dev).to(torch.int16)
    rfi[torch.rand(at // cols, generator=g, device=dev) < 0.03] = -797           # (what a row of zeros has)
    cfi = torch.randint(-8, 9, (cols * len(sizes),), generator=g, device=dev).to(torch.int16)
    scl = torch.randint(0, 16, (cols * len(sizes),), generator=g, device=dev).to(torch.int8)
    none = torch.zeros(1, dtype=torch.int32, device=dev)
    side = (p(rfi), p(cfi), p(scl), p(none))
    ntab = 656 * (int(roles.max()) + 1)
    counts = torch.zeros(ntab * 256, dtype=torch.int32, device=dev)
    call("sg_r2_hist", p(w), p(tb), p(sg), nseg, *side, p(counts))
    assert int(counts.sum()) == 3 * int(ns.sum())
    freq, used = normalize(counts.cpu().numpy().reshape(ntab, 256), 1 << 15)
    full = np.zeros((ntab, 256), np.uint16)
    full[used] = freq
    if extra is not None:
        row = full[512 + np.flatnonzero(full[512:640].any(1))[0]]
        row[int(row.argmax())] -= 5
        row[extra] = 5
    f = torch.from_numpy(full.view(np.int16)).cuda()
    enc, lut = torch.empty(ntab * 512, dtype=torch.int32, device=dev), torch.empty(ntab * 1280, dtype=torch.uint8, device=dev)
    call("sg_rans_tables", p(f), ntab, 15, p(enc), p(lut))
    cap = 1024
    slots, lens = torch.empty(nseg * cap, dtype=torch.uint8, device=dev), torch.empty(nseg, dtype=torch.int32, device=dev)
    call("sg_r2_encode", p(w), p(tb), p(sg), nseg, *side, p(enc), p(slots), cap, p(lens))
    total = int(lens.sum(dtype=torch.int64))
    assert int(lens.min()) >= 4 and total < nseg * cap
    stream, off = torch.zeros((total + 31) // 16 * 16, dtype=torch.uint8, device=dev), torch.empty(nseg + 1, dtype=torch.int64, device=dev)
    call("sg_scan_gather", p(slots), cap, p(lens), nseg, p(stream), total, p(off))
    back = torch.full_like(w, -1)
    call("sg_r2_decode", p(stream), p(off), p(off[1:]), p(back), p(tb), p(sg), nseg, *side, p(enc), p(lut))
    bits = ctypes.c_int(0)
    _lib.check(L.sg_status_fetch(0, st, ctypes.byref(bits)), "sg_status_fetch")
    coded = torch.zeros(at, dtype=torch.bool, device=dev)                        # (a tensor's last row may reach past its segments)
    for r, k in zip(rowbase, sizes):
        coded[int(r) * cols:int(r) * cols + int(k)] = True
    assert bits.value == 0 and torch.equal(back[coded], w[coded]) and bool((back[~coded] == -1).all())
