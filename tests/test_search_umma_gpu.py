"""The search whose scores come from the tensor cores against the oracle's scan: token counts around its tiles of 128, runs
of one tile and of many, and columns and rows whose scores decide little or nothing - ties, several magnitudes within one
CTA, more undecided tokens than a warp's queue holds, overflow, infinities and NaN.  Indices are compared exactly."""
import numpy as np
import pytest

import oracle
import pim_dl_asplos_b200 as P  # noqa: F401

pytestmark = pytest.mark.gpu

FEWEST = 96000000   # scores from which on a call takes this form


def _inputs(v, CT, CB, M, mixed):
    rng = np.random.default_rng(v * 1000 + CT + mixed)
    x = rng.standard_normal((M, CB, v), dtype=np.float32)
    cen = rng.standard_normal((CB, CT, v), dtype=np.float32)
    if mixed:
        x[::5] = np.round(x[::5] * 2) / 2                       # ties with the rounded codebooks
        x[1::5] *= np.exp2(rng.integers(-30, 30, (x[1::5].shape[0], 1, 1))).astype(np.float32)
        x[2::15, rng.integers(0, CB)] = np.nan
        x[7::15, rng.integers(0, CB)] = np.inf
        x[12::1000] = 1e25
        cen[1::8] = np.round(cen[1::8] * 2) / 2
        cen[2::8] *= 1e-3
        cen[3::8, ::2] *= 1e3
        cen[4::8, 1] = cen[4::8, 0]                             # twins: every token next to them is undecided
        cen[5::8, CT // 2] = np.inf
        cen[6::8, CT - 1] = np.nan
        cen[7::8, :, 0] = 1e19
    return np.ascontiguousarray(x.reshape(M, CB * v)), np.ascontiguousarray(cen)


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("v,CT,CB,over", [(2, 32, 8, 0), (4, 32, 16, 1), (4, 64, 8, 127), (4, 64, 192, 63), (4, 128, 4, 1),
                                          (8, 32, 6, 64), (8, 64, 96, 129)])
def test_indices_equal_the_scan(ctx, v, CT, CB, over, mixed):
    import torch
    M = -(-FEWEST // (CB * CT) // 128) * 128 + 128 + over
    x, cen = _inputs(v, CT, CB, M, mixed)
    ctx.load_weights(78, cen, np.zeros((CB, CT, 16), np.int8), np.zeros(16, np.float32), 1.0)
    with np.errstate(all="ignore"):
        want = oracle.index_calculation(x, cen).astype(np.uint8)
    idx = torch.full((M + 1, CB), 255, dtype=torch.uint8, device="cuda")
    xd = torch.from_numpy(x).cuda()
    torch.cuda.synchronize()
    ctx.index_calculation(78, xd, idx[:M])
    got = idx.cpu().numpy()
    assert np.array_equal(got[:M], want)
    assert (got[M] == 255).all()
    ctx.unload_weights(78)


def test_every_token_undecided(ctx):
    """All centroids alike: the queue overflows in every tile, and the scan keeps the first."""
    import torch
    v, CT, CB, M = 4, 64, 8, FEWEST // 512 + 77
    ctx.load_weights(79, np.ones((CB, CT, v), np.float32), np.zeros((CB, CT, 16), np.int8), np.zeros(16, np.float32), 1.0)
    idx = torch.full((M, CB), 255, dtype=torch.uint8, device="cuda")
    x = torch.randn(M, CB * v, device="cuda")
    torch.cuda.synchronize()
    ctx.index_calculation(79, x, idx)
    assert not idx.any()
    ctx.unload_weights(79)
