"""The encoder layer's replayed forward gives the bytes of the ordinary one, a tensor of its own per call, and follows
weights and plans that change between calls."""
import numpy as np
import pytest

import pim_dl_asplos_b200 as P
from pim_dl_asplos_b200 import layer as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("separate_qkv", [False, True])
def test_replayed_forward(ctx, separate_qkv):
    import torch
    S, B, H, D, F = 19, 3, 4, 64, 256
    cb = {"qkv": 32, "o": 32, "ffn1": 32, "ffn2": 128}
    w = L.random_layer_weights(D, F, cb, {k: 16 for k in cb}, seed=9, separate_qkv=separate_qkv)
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    lay = L.LutTransformerLayer(ctx, w, S, B, H, first_layer_id=60)
    xs = [torch.from_numpy(L.synth.make_input(S * B, D, seed=i)).cuda() for i in range(3)]
    torch.cuda.synchronize()

    def plain(x):
        h, f = lay._body(x)
        return h + f

    with torch.cuda.stream(stream):
        want = [plain(x) for x in xs]
        got = [lay.forward(xs[i % 3]) for i in range(12)]
        stream.synchronize()
        assert lay._graph is not None
        for i, y in enumerate(got):
            assert torch.equal(y, want[i % 3])
        assert len({y.data_ptr() for y in got}) == 12
        # other weights behind the same layer id: the captured forward must not be used
        cen, lut, bias, scale, lut_bias = w["o"]
        ctx.load_weights(lay.ids["o"], cen, np.roll(lut, 1, axis=2), bias, scale, lut_bias)
        want = [plain(x) for x in xs]
        got = [lay.forward(xs[i % 3]) for i in range(9)]
        stream.synchronize()
        for i, y in enumerate(got):
            assert torch.equal(y, want[i % 3])
        # scratch that grows moves: a large call in between
        big = 70
        ctx.load_weights(big, np.zeros((512, 16, 2), np.float32), np.zeros((512, 16, 64), np.int8), np.zeros(64, np.float32), 1.0)
        xb, yb = torch.zeros(9000, 1024, device="cuda"), torch.empty(9000, 64, device="cuda")
        ctx.amm_host(big, xb, yb, flags=P.FLAG_ASYNC)
        got = [lay.forward(xs[i % 3]) for i in range(9)]
        stream.synchronize()
        for i, y in enumerate(got):
            assert torch.equal(y, want[i % 3])
    ctx.set_stream(None)
    for lid in list(lay.ids.values()) + [big]:
        ctx.unload_weights(lid)
