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
