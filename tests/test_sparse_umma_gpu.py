"""The sparse tcgen05 kernel (CTA pairs) against the oracle at the edges of its tiles: row tiles of 256 split over two
CTAs, column tiles that N does not divide, every centroid count (each packs its operand its own way), half-filled last
slabs, several tiles per pair, out-of-range indices and the fused activation."""
import numpy as np
import pytest

import oracle
import pim_dl_asplos_b200 as P

pytestmark = pytest.mark.gpu

#        M     CB  CT   N
SHAPES = [(1, 16, 16, 16), (128, 16, 8, 64), (129, 48, 8, 144), (256, 16, 32, 160), (257, 32, 16, 176), (130, 16, 64, 336),
          (385, 16, 128, 80), (70, 16, 256, 320), (3000, 32, 16, 1040), (5000, 16, 8, 1600)]


@pytest.mark.parametrize("n_tile", [0, 64, 128, 160])
@pytest.mark.parametrize("M,CB,CT,N", SHAPES)
def test_sparse_form(ctx, M, CB, CT, N, n_tile):
    rng = np.random.default_rng(M + CB + CT + N)
    cen = rng.standard_normal((CB, CT, 2), dtype=np.float32)
    lut = rng.integers(-128, 128, (CB, CT, N), dtype=np.int8)
    bias = rng.standard_normal(N, dtype=np.float32)
    idx = rng.integers(0, CT, (M, CB), dtype=np.uint8)
    ctx.load_weights(78, cen, lut, bias, 0.013, 0.3)
    ctx.set_plan(78, variant=P.VARIANT_UMMA, umma_operand=3, umma_n_tile=n_tile)
    acc = oracle.lut_gather(idx.astype(np.uint16), lut)
    want = oracle.dequant(acc, bias, CB, 0.013, 0.3)
    y = np.zeros((M, N), np.float32)
    for _ in range(2):
        ctx.pim_lut(78, idx, y)
        assert np.array_equal(y.view(np.uint32), want.view(np.uint32))
        y[:] = 0
    if CT < 256:   # an index beyond the table adds nothing
        beyond = rng.random((M, CB)) < 0.1
        acc = sum(np.where(beyond[:, c, None], 0, lut[c, idx[:, c]].astype(np.int32)) for c in range(CB))
        want = oracle.dequant(np.ascontiguousarray(acc, np.int32), bias, CB, 0.013, 0.3)
        idx = np.where(beyond, rng.integers(CT, 256, (M, CB)), idx).astype(np.uint8)
        ctx.pim_lut(78, idx, y)
        assert np.array_equal(y.view(np.uint32), want.view(np.uint32))
    ctx.set_activation(78, P.ACT_GELU_TANH)
    ctx.pim_lut(78, idx, y)
    np.testing.assert_allclose(y, oracle.gelu_tanh(want), rtol=1e-5, atol=1e-9)
    ctx.unload_weights(78)


@pytest.mark.parametrize("n_tile,split", [(0, 0), (64, 2), (64, 5), (64, 16), (128, 3), (128, 9)])
@pytest.mark.parametrize("M,CB,CT,N", [(1, 512, 16, 64), (130, 1536, 16, 80), (300, 96, 64, 144), (60, 96, 256, 96), (40, 464, 8, 64)])
def test_split_codebook_axis(ctx, M, CB, CT, N, n_tile, split):
    """Slices of one tile on several pairs, summed through scratch; twice, so that the counters have been re-armed."""
    rng = np.random.default_rng(M + CB + N)
    lut = rng.integers(-128, 128, (CB, CT, N), dtype=np.int8)
    bias = rng.standard_normal(N, dtype=np.float32)
    idx = rng.integers(0, CT, (M, CB), dtype=np.uint8)
    ctx.load_weights(79, rng.standard_normal((CB, CT, 1), dtype=np.float32), lut, bias, 0.013, 0.3)
    ctx.set_plan(79, variant=P.VARIANT_UMMA, umma_operand=3 if n_tile else 0, umma_n_tile=n_tile, umma_split=split)
    want = oracle.dequant(oracle.lut_gather(idx.astype(np.uint16), lut), bias, CB, 0.013, 0.3)
    for _ in range(2):
        y = np.full((M, N), np.nan, np.float32)
        ctx.pim_lut(79, idx, y)
        assert np.array_equal(y.view(np.uint32), want.view(np.uint32))
    ctx.set_activation(79, P.ACT_GELU_TANH)
    ctx.pim_lut(79, idx, y)
    np.testing.assert_allclose(y, oracle.gelu_tanh(want), rtol=1e-5, atol=1e-9)
    ctx.unload_weights(79)


@pytest.mark.parametrize("M,CB,CT,N", [(1024, 16, 16, 3312), (1000, 48, 8, 3072), (300, 32, 32, 6160), (2049, 16, 64, 1536), (1024, 16, 256, 3280)])
def test_one_wide_tile_per_pair(ctx, M, CB, CT, N):
    """Where 192-column tiles make one round of what narrower ones would make two the default plan takes them; N that 192
    and 32 do not divide, rows past M, and the fused activation."""
    rng = np.random.default_rng(M + N)
    cen = rng.standard_normal((CB, CT, 2), dtype=np.float32)
    lut = rng.integers(-128, 128, (CB, CT, N), dtype=np.int8)
    bias = rng.standard_normal(N, dtype=np.float32)
    idx = rng.integers(0, CT, (M, CB), dtype=np.uint8)
    ctx.load_weights(79, cen, lut, bias, 0.013, 0.3)
    want = oracle.dequant(oracle.lut_gather(idx.astype(np.uint16), lut), bias, CB, 0.013, 0.3)
    for _ in range(2):
        y = np.zeros((M, N), np.float32)
        ctx.pim_lut(79, idx, y)
        assert np.array_equal(y.view(np.uint32), want.view(np.uint32))
    ctx.set_activation(79, P.ACT_GELU_TANH)
    ctx.pim_lut(79, idx, y)
    np.testing.assert_allclose(y, oracle.gelu_tanh(want), rtol=1e-5, atol=1e-9)
    ctx.unload_weights(79)
