"""Dequantisers of the 20 types that archives hold, in NumPy from the layouts of the blocks (ggml-common.h's block_<type>,
ggml-quants.c's dequantize_row_<type>): float32 operations one by one in the order of those functions."""
import numpy as np

F = np.float32
KV = np.array([-127, -104, -83, -65, -49, -35, -22, -10, 1, 13, 25, 38, 53, 69, 89, 113], np.float32)      # the IQ4 levels
GRID = {16: 0, 17: 1, 19: 2, 29: 2, 22: 3, 18: 4, 21: 5}                                                    # type -> lattice table


def _f16(b):
    """two bytes of every block as float32, one column"""
    return np.ascontiguousarray(b).view(np.float16).astype(F)


def _k4(b):
    """the 8 six-bit scales and mins of Q4_K / Q5_K"""
    lo, mid, hi = b[:, 0:4].astype(int), b[:, 4:8].astype(int), b[:, 8:12].astype(int)
    sc = np.concatenate([lo & 63, (hi & 15) | (lo >> 6) << 4], 1)
    mn = np.concatenate([mid & 63, (hi >> 4) | (mid >> 6) << 4], 1)
    return sc.astype(F), mn.astype(F)


def _points(t, idx):
    """lattice points idx [blocks][groups] -> their values, one weight each"""
    from seedpack_b200 import tables
    grid = tables.host(GRID[t], 0)
    lev = (grid.view(np.uint8).reshape(len(grid), -1).astype(int) - 1) // 2        # the tables hold 2 level + 1
    if t in (16, 17, 22):
        lev = np.array([8, 25, 43])[lev]
    elif t == 18:
        lev = np.where(lev == 7, 62, 4 + 8 * lev)
    elif t == 21:
        lev = 2 * lev + 1
    else:
        lev = lev - 1
    return lev.astype(F)[idx].reshape(len(idx), 256)


def _signs7(s):
    """seven stored sign bits [blocks][units] and the one that makes the minuses even -> +-1 per weight"""
    bits = (s[:, :, None] >> np.arange(7)) & 1
    bits = np.concatenate([bits, bits.sum(2, keepdims=True) & 1], 2)
    return np.where(bits, F(-1), F(1)).reshape(len(s), 256)


def dequantize(t, y, bs):
    """y: uint8 blocks of type t back to back -> float32 [blocks][weights per block]"""
    b = y.reshape(-1, bs)
    n = len(b)
    with np.errstate(all="ignore"):
        if t in (2, 3, 6, 7):
            d, o = _f16(b[:, :2]), 2
            if t in (3, 7):
                m, o = _f16(b[:, 2:4]), 4
            hi = 0
            if t in (6, 7):
                hi = np.unpackbits(b[:, o:o + 4], axis=1, bitorder="little").astype(int) << 4
                o += 4
            q = np.concatenate([b[:, o:] & 15, b[:, o:] >> 4], 1).astype(int) | hi
            return q.astype(F) * d + m if t in (3, 7) else (q - (8 if t == 2 else 16)).astype(F) * d
        if t == 8:
            return b[:, 2:].view(np.int8).astype(F) * _f16(b[:, :2])
        if t == 42:
            q = (b[:, 2:, None] >> (2 * np.arange(4))) & 3
            return (q.reshape(n, 64).astype(int) - 1).astype(F) * _f16(b[:, :2])
        w = np.arange(256)
        two = lambda qs: (qs[:, 32 * (w // 128) + w % 32] >> (2 * (w % 128 // 32))) & 3                      # 2-bit planes of 32 weights
        if t == 10:
            sc = b[:, w // 16]
            return _f16(b[:, 80:82]) * (sc & 15).astype(F) * two(b[:, 16:80]).astype(F) - _f16(b[:, 82:84]) * (sc >> 4).astype(F)
        if t == 11:
            h = (b[:, w % 32] >> (4 * (w // 128) + w % 128 // 32)) & 1
            s, a = np.arange(16), b[:, 96:108].astype(int)
            sc = ((np.where(s < 8, a[:, s % 8] & 15, a[:, s % 8] >> 4)) | ((a[:, 8 + s % 4] >> (2 * (s // 4))) & 3) << 4) - 32
            return _f16(b[:, 108:110]) * sc[:, w // 16].astype(F) * ((two(b[:, 32:96]) | h << 2).astype(int) - 4).astype(F)
        if t in (12, 13):
            sc, mn = _k4(b[:, 4:16])
            qs = b[:, 48:] if t == 13 else b[:, 16:]
            q = (qs[:, 32 * (w // 64) + w % 32] >> (4 * (w % 64 // 32))) & 15
            if t == 13:
                q = q | ((b[:, 16 + w % 32] >> (w // 32)) & 1) << 4
            return _f16(b[:, :2]) * sc[:, w // 32] * q.astype(F) - _f16(b[:, 2:4]) * mn[:, w // 32]
        if t == 14:
            j = w % 128 // 32
            q = ((b[:, 64 * (w // 128) + 32 * (j & 1) + w % 32] >> (4 * (j >> 1))) & 15) | ((b[:, 128 + 32 * (w // 128) + w % 32] >> (2 * j)) & 3) << 4
            return _f16(b[:, 208:210]) * b[:, 192:208].view(np.int8)[:, w // 16].astype(F) * (q.astype(int) - 32).astype(F)
        if t == 20:
            return _f16(b[:, :2]) * KV[np.concatenate([b[:, 2:] & 15, b[:, 2:] >> 4], 1)]
        if t == 23:
            sh, s = np.ascontiguousarray(b[:, 2:4]).view(np.uint16).astype(int), np.arange(8)
            ls = (((b[:, 4 + s // 2] >> (4 * (s % 2))) & 15).astype(int) | ((sh >> (2 * s)) & 3) << 4) - 32
            q = (b[:, 8 + 16 * (w // 32) + w % 16] >> (4 * (w % 32 // 16))) & 15
            return _f16(b[:, :2]) * ls[:, w // 32].astype(F) * KV[q]
        u, g = np.arange(32), np.arange(64)
        if t == 16:
            a = np.ascontiguousarray(b[:, 2:66]).view(np.uint32).reshape(n, 8, 2)
            aux = a[:, :, 1]
            s7 = ((aux[:, u // 4] >> (7 * (u % 4)).astype(np.uint32)) & 127).astype(int)
            db = _f16(b[:, :2]) * (F(0.5) + (aux >> 28).astype(F)) * F(0.25)
            return db[:, w // 32] * _points(t, b[:, 2 + 8 * (u // 4) + u % 4]) * _signs7(s7)
        if t == 17:
            qs = np.ascontiguousarray(b[:, 2:66]).view(np.uint16).astype(int)
            nib = (b[:, 66 + w // 32] >> (4 * (w // 16 % 2))) & 15
            return _f16(b[:, :2]) * (F(0.5) + nib.astype(F)) * F(0.25) * _points(t, qs & 511) * _signs7(qs >> 9)
        if t == 18:
            aux = np.ascontiguousarray(b[:, 66:98]).view(np.uint32)
            s7 = ((aux[:, u // 4] >> (7 * (u % 4)).astype(np.uint32)) & 127).astype(int)
            db = _f16(b[:, :2]) * (F(0.5) + (aux >> 28).astype(F)) * F(0.5)
            return db[:, w // 32] * _points(t, b[:, 2:66]) * _signs7(s7)
        if t == 19:
            qh = np.ascontiguousarray(b[:, 34:50]).view(np.uint16).astype(int)
            idx = b[:, 2:34].astype(int) | ((qh[:, u // 4] >> (3 * (u % 4))) & 7) << 8
            dl = _f16(b[:, :2]) * (2 * ((qh >> 12) & 7) + 1).astype(F)
            delta = np.where(qh & 0x8000, F(-0.125), F(0.125))
            return dl[:, w // 32] * (_points(t, idx) + delta[:, w // 32])
        sign = lambda o: np.where(np.unpackbits(b[:, o:o + 32], axis=1, bitorder="little"), F(-1), F(1))
        if t == 21:
            idx = b[:, 2:66].astype(int) | ((b[:, 66 + g // 8] >> (g % 8)) & 1).astype(int) << 8
            nib = (b[:, 106 + w // 64] >> (4 * (w // 32 % 2))) & 15
            return _f16(b[:, :2]) * (1 + 2 * nib.astype(int)).astype(F) * _points(t, idx) * sign(74)
        if t == 22:
            idx = b[:, 2:34].astype(int) | ((b[:, 66 + u // 4] >> (2 * (u % 4))) & 3).astype(int) << 8
            nib = (b[:, 74 + w // 32] >> (4 * (w // 16 % 2))) & 15
            return _f16(b[:, :2]) * (F(0.5) + nib.astype(F)) * F(0.25) * _points(t, idx) * sign(34)
        assert t == 29
        sc = np.ascontiguousarray(b[:, 48:56]).view(np.uint16).astype(int)
        d = (sc[:, 0] >> 12) | ((sc[:, 1] >> 8) & 0xf0) | ((sc[:, 2] >> 4) & 0xf00) | (sc[:, 3] & 0xf000)
        d = d.astype(np.uint16).view(np.float16).astype(F)[:, None]
        qh = b[:, 32 + u // 2].astype(int) >> (4 * (u % 2))
        idx = b[:, :32].astype(int) | (qh & 7) << 8
        dl = d * (2 * ((sc[:, w // 64] >> (3 * (w // 16 % 4))) & 7) + 1).astype(F)
        return dl * (_points(t, idx) + np.where(qh & 8, F(-0.125), F(0.125))[:, w // 8])
