"""Few tokens: the kernel that reads only the used rows of the table, which the library chooses by itself, against the
oracle: shares of the codebook axis that do not divide it, more codebooks than one int32 sum takes, ragged column tiles,
any centroid count, out-of-range indices, the fused activation, and the call that allocates nothing."""
import ctypes

import numpy as np
import pytest

import oracle
import pim_dl_asplos_b200 as P
from pim_dl_asplos_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,CB,CT,N", [(1, 1, 16, 16), (1, 1000, 16, 144), (2, 77, 13, 272), (3, 2600, 16, 128), (5, 64, 256, 1040), (16, 96, 16, 2000),
                                       (33, 384, 16, 96), (40, 48, 200, 3056),
                                       # shares of 8 and more chunks of 256 codebooks: sums of 16 bits as full as they get
                                       (600, 4096, 13, 16), (600, 4098, 13, 16), (600, 4610, 13, 32), (2, 17000, 13, 16), (260, 511, 13, 144)])
def test_rows(ctx, M, CB, CT, N):
    rng = np.random.default_rng(M + CB + CT + N)
    cen = rng.standard_normal((CB, CT, 2), dtype=np.float32)
    lut = rng.integers(-128, 128, (CB, CT, N), dtype=np.int8)
    lut[:, 0] = -128
    lut[:, 1] = 127
    bias = rng.standard_normal(N, dtype=np.float32)
    idx = rng.integers(0, CT, (M, CB), dtype=np.uint8)
    idx[0] = 1
    idx[-1] = 0
    ctx.load_weights(81, cen, lut, bias, 0.013, 0.3)
    y = np.zeros((M, N), np.float32)
    ctx.pim_lut(81, idx, y)
    want = oracle.dequant(oracle.lut_gather(idx.astype(np.uint16), lut), bias, CB, 0.013, 0.3)
    assert np.array_equal(y.view(np.uint32), want.view(np.uint32))
    if CT < 256:   # an index beyond the table adds nothing
        beyond = rng.random((M, CB)) < 0.2
        acc = sum(np.where(beyond[:, c, None], 0, lut[c, idx[:, c]].astype(np.int32)) for c in range(CB))
        want = oracle.dequant(np.ascontiguousarray(acc, np.int32), bias, CB, 0.013, 0.3)
        ctx.pim_lut(81, np.where(beyond, rng.integers(CT, 256, (M, CB)), idx).astype(np.uint8), y)
        assert np.array_equal(y.view(np.uint32), want.view(np.uint32))
    ctx.set_activation(81, P.ACT_GELU_TANH)
    ctx.pim_lut(81, idx, y)
    want = oracle.dequant(oracle.lut_gather(idx.astype(np.uint16), lut), bias, CB, 0.013, 0.3)
    np.testing.assert_allclose(y, oracle.gelu_tanh(want), rtol=1e-5, atol=1e-9)
    ctx.unload_weights(81)


@pytest.mark.parametrize("offset", [0, 4])
def test_static_scratch_rows(offset):
    """... and a table that is not 16-byte aligned, which goes another way."""
    import torch
    M, K, N = 3, 512, 1040
    c = synth.make_case(M=M, K=K, N=N, v=2, CT=16, seed=3)
    x, cen, bias = (torch.from_numpy(a).cuda() for a in (c.x, c.centroid, c.bias))
    room = torch.empty(c.lut.size + 16, dtype=torch.int8, device="cuda")
    room[offset:offset + c.lut.size] = torch.from_numpy(c.lut).cuda().reshape(-1)
    y = torch.full((M, N), float("nan"), device="cuda")
    torch.cuda.synchronize()
    ip, lp = P.make_params(M, K, N, K // 2, 16, c.scale, c.lut_bias)
    rc = P.load_library().lutamm_amm_static_scratch(0, None, x.data_ptr(), cen.data_ptr(), room.data_ptr() + offset, bias.data_ptr(), y.data_ptr(),
                                                    ctypes.byref(ip), ctypes.byref(lp))
    assert rc == P.OK
    want = oracle.amm(c.x, c.centroid, c.lut, c.bias, c.scale, c.lut_bias)[0]
    assert np.array_equal(y.cpu().numpy().view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("M,K,N,v,CT", [(1, 768, 768, 2, 16), (3, 512, 144, 4, 8), (2, 320, 48, 8, 13), (1, 2080, 16, 2, 64), (1, 4400, 272, 8, 4), (1, 12, 32, 4, 31)])
def test_search_and_rows_in_one_launch(ctx, M, K, N, v, CT):
    """Ties and near-ties, which the order of the scan decides, and values that do not compare."""
    rng = np.random.default_rng(K + N)
    cen = (rng.integers(-3, 4, (K // v, CT, v)) * 0.5).astype(np.float32)
    x = (rng.integers(-3, 4, (M, K)) * 0.5).astype(np.float32)
    x[:, ::3] += rng.normal(0, 3e-7, x[:, ::3].shape).astype(np.float32)
    x[0, -1] = np.nan
    lut = rng.integers(-128, 128, (K // v, CT, N), dtype=np.int8)
    bias = rng.standard_normal(N, dtype=np.float32)
    import torch
    ctx.load_weights(82, cen, lut, bias, 0.02, -0.4)
    y = torch.full((M, N), float("nan"), device="cuda")
    xd = torch.from_numpy(x).cuda()
    torch.cuda.synchronize()
    ctx.amm_host(82, xd, y)
    want = oracle.amm(x, cen, lut, bias, 0.02, -0.4)[0]
    assert np.array_equal(y.cpu().numpy().view(np.uint32), want.view(np.uint32))
    ctx.unload_weights(82)
