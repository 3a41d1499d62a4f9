"""When a layer's captured forward may be replayed: a set-up that changes between calls takes the ordinary path again.  On
the CPU, with a graph that records nothing and a context that only has what the key is made of."""
import types

import pytest
import torch

import pim_dl_asplos_b200 as P
from pim_dl_asplos_b200 import layer as L


class _Graph:
    def capture_begin(self, **kw):
        pass

    def capture_end(self):
        pass

    def replay(self):
        self.replayed = True


class _Torch:
    """torch, with a stream and graphs that need no GPU."""
    cuda = types.SimpleNamespace(current_stream=lambda device: types.SimpleNamespace(cuda_stream=7), is_current_stream_capturing=lambda: False,
                                 CUDAGraph=_Graph)

    def __getattr__(self, name):
        return getattr(torch, name)


class _Library:
    queued = 0

    def lutamm_launch_count(self, handle):
        return self.queued


class _Context(P.LutAmmContext):
    generation = 1

    def __init__(self):
        self._L, self._h, self.device, self.stream = _Library(), None, None, 7


class _Layer(L.LutTransformerLayer):
    def __init__(self, n=4, dim=8):
        self.ctx = _Context()
        self.torch, self.n, self.token_dim, self.fused_gelu, self.ln = _Torch(), n, dim, True, {"ln1": (torch.ones(dim), torch.zeros(dim))}
        self._graph, self._seen, self._seen_key = None, 0, None
        self.bodies = 0

    def _body(self, x):
        self.bodies += 1
        self.ctx._L.queued += 8
        return x + 1, 2 * x


def _captured(lay, x):
    for _ in range(4):
        lay.forward(x)
    assert lay._graph is not None and lay._graph[1].replayed
    lay.bodies = 0
    return lay


def test_a_forward_captured_in_inference_mode_is_not_replayed_outside():
    x = torch.arange(32.0).view(4, 8)
    with torch.inference_mode():
        lay = _captured(_Layer(), x)
    y = lay.forward(x)
    assert lay.bodies == 1 and torch.equal(y, 3 * x + 1)
    lay = _captured(_Layer(), x)
    with torch.inference_mode():
        assert torch.equal(lay.forward(x), 3 * x + 1)


@pytest.mark.parametrize("owner", [torch.backends.cuda.matmul, torch.backends])
def test_either_api_of_the_matmul_precision(owner):
    """Reading allow_tf32 raises once a program has set fp32_precision.  The precision itself belongs to what a capture is
    valid for: attention by two matrix products follows it."""
    x = torch.ones(4, 8)
    before = owner.fp32_precision
    lay = _captured(_Layer(), x)
    try:
        owner.fp32_precision = "tf32"
        assert torch.equal(lay.forward(x), 3 * x + 1) and lay.bodies == 1
    finally:
        owner.fp32_precision = before


def test_the_priority_of_the_attention_back_ends():
    from torch.nn.attention import SDPBackend, sdpa_kernel
    every = [SDPBackend.MATH, SDPBackend.EFFICIENT_ATTENTION, SDPBackend.FLASH_ATTENTION, SDPBackend.CUDNN_ATTENTION]
    x = torch.ones(4, 8)
    lay = _Layer()
    with sdpa_kernel(every, set_priority=True):
        _captured(lay, x)
    with sdpa_kernel(every[::-1], set_priority=True):
        lay.forward(x)
    assert lay.bodies == 1


def test_no_branch_for_a_replaced_operator_call():
    """Whether a forward may be replayed does not depend on how a test watches its linears."""
    lay, x = _Layer(), torch.ones(4, 8)
    key = lay._graph_key(x)
    lay._amm = None
    assert key is not None and lay._graph_key(x) == key


def test_launches_of_a_replayed_forward_count():
    """Each forward runs eight kernels of the library, whether it queues them or replays them; recording them runs none."""
    lay, x = _Layer(), torch.ones(4, 8)
    for forwards in range(1, 9):
        lay.forward(x)
        assert lay.ctx.launch_count == 8 * forwards
    assert lay._graph[1].replayed


def test_what_the_ordinary_call_refuses_or_autograd_follows_is_not_replayed():
    import torch.autograd.forward_ad as fw
    x = torch.ones(4, 8)
    lay = _captured(_Layer(), x)
    assert lay._graph_key(torch.ones(8, 4).t()) is None           # the operator takes contiguous tensors only
    with fw.dual_level():                                       # the addition of x carries its tangent
        assert lay._graph_key(fw.make_dual(x, x)) is None
        assert lay._graph_key(x) is not None

    class Tensor(torch.Tensor):
        pass

    assert lay._graph_key(x.as_subclass(Tensor)) is None
    lay.ln["ln1"][0].requires_grad_()
    assert lay._graph_key(x) is None
    with torch.no_grad():
        assert lay._graph_key(x) is not None


@pytest.mark.gpu
def test_replayed_forward_in_and_out_of_inference_mode(ctx):
    """The layer itself on the GPU: the same bytes in every mode, and its launches counted in each."""
    S, B, H, D, F = 16, 2, 4, 64, 128
    cb = {"qkv": 32, "o": 32, "ffn1": 32, "ffn2": 64}
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    lay = L.LutTransformerLayer(ctx, L.random_layer_weights(D, F, cb, {k: 16 for k in cb}, seed=4), S, B, H, first_layer_id=84)
    x = torch.from_numpy(L.synth.make_input(S * B, D, seed=4)).cuda()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        want = torch.add(*lay._body(x))
        for mode in (torch.inference_mode, torch.no_grad, torch.enable_grad):
            lay.forward(x)
            before = ctx.launch_count
            lay.forward(x)
            ordinary = ctx.launch_count - before
            with mode():
                for _ in range(5):
                    before = ctx.launch_count
                    assert torch.equal(lay.forward(x), want)
                    assert ctx.launch_count - before == ordinary > 0
            assert lay._graph is not None
        stream.synchronize()
    ctx.set_stream(None)
    for lid in lay.ids.values():
        ctx.unload_weights(lid)
