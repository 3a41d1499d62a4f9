"""The search kernels' filter against the oracle's scan, where the two could part: near-ties and exact ties,
magnitudes at which 1e-6 is everything or nothing, overflow and NaN, and the edges of both kernels' tiles
(codebook blocks, token blocks of one and two per thread, padded centroid groups, unaligned activations)."""
import numpy as np
import pytest

import oracle
import pim_dl_asplos_b200 as P  # noqa: F401

pytestmark = pytest.mark.gpu

SHAPES = [(2, 8, 3, 5), (2, 16, 130, 515), (2, 32, 17, 257), (4, 8, 33, 129), (4, 64, 9, 300), (4, 128, 4, 128), (1, 5, 40, 70),
          (3, 17, 7, 131), (8, 16, 5, 513), (10, 16, 6, 64), (12, 16, 5, 90), (16, 13, 3, 140), (20, 256, 3, 33), (32, 16, 2, 200)]


@pytest.mark.parametrize("data", ["normal", "ties", "tiny", "large", "overflow", "nonfinite"])
@pytest.mark.parametrize("v,CT,CB,M", SHAPES)
def test_indices_equal_the_scan(ctx, v, CT, CB, M, data):
    import torch
    rng = np.random.default_rng(v * 1000 + CT)
    x = rng.standard_normal((M, CB * v), dtype=np.float32)
    cen = rng.standard_normal((CB, CT, v), dtype=np.float32)
    if data == "ties":
        x, cen = np.round(x * 2) / 2, np.round(cen * 2) / 2
    elif data != "normal":
        f = np.float32({"tiny": 1e-3, "large": 1e4, "overflow": 1e19, "nonfinite": 1}[data])
        x, cen = x * f, cen * f
    if data == "nonfinite":
        for a in (x, cen):
            a[rng.random(a.shape) < 0.02] = np.nan
            a[rng.random(a.shape) < 0.02] = np.inf
    x, cen = np.ascontiguousarray(x, np.float32), np.ascontiguousarray(cen, np.float32)
    ctx.load_weights(77, cen, np.zeros((CB, CT, 16), np.int8), np.zeros(16, np.float32), 1.0)
    with np.errstate(all="ignore"):
        want = oracle.index_calculation(x, cen).astype(np.uint8)
    for offset in (0, 1):   # floats past a 16-byte boundary
        buf = torch.zeros(M * CB * v + 4, device="cuda")
        xd = buf[offset:offset + x.size].view(M, CB * v)
        xd.copy_(torch.from_numpy(x))
        idx = torch.full((M, CB), 255, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        ctx.index_calculation(77, xd, idx)
        assert np.array_equal(idx.cpu().numpy(), want)
    ctx.unload_weights(77)
