"""Performance cases of the LUT-AMM operator and its callers.

What a user of this package has it do, through its public entry points:

  amm      one linear on device buffers, queued asynchronously (lutamm_amm / amm_host)
  linears  the four linears of an encoder layer back to back, as bench.py steps through them
  layer    LutTransformerLayer.forward: the four linears with attention, LayerNorm, GELU and residuals
  host     the four linears through pinned host buffers, one lutamm_sync at the end
  static   lutamm_amm_static_scratch, the call that allocates nothing
  build    build_lut, the int8 table of a linear from its centroids and dense weight (checkpoint conversion)

Shapes are those of the package's configurations (inference_engine/configs, run_experiments.py, synth.WORKLOADS).
Every output is compared exactly: indices and int32 sums are whole numbers, the dequantisation is a stated
sequence of roundings, and a layer feeds each linear's float output to the next linear's nearest-centroid search,
where one bit may select another table row."""
import ctypes
import itertools
import math

import torch

import pim_dl_asplos_b200 as P
from pim_dl_asplos_b200 import layer as L


def _case(name, kind, **kw):
    c = dict(kind=kind, v=2, CT=16, scale=0.01, lut_bias=0.0)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one short request (32 tokens) through an attention-output linear: nothing but latency and launches
        _case("amm_o_32", "amm", M=32, K=768, N=768),
        # configs/bert_base_ffn1_amm.yaml: 4 sequences of 128 tokens through FFN1
        _case("amm_ffn1_512", "amm", M=512, K=768, N=3072),
        # one sequence through a whole BERT-base layer: online inference
        _case("layer_base_1x128", "layer", batch=1, seq=128, D=768, F=3072, heads=12),
        # configs/bert_large_layer.yaml: a batch of 16 full-length sequences through a BERT-large layer
        _case("layer_large_16x512", "layer", batch=16, seq=512, D=1024, F=4096, heads=16, v=4),
        # configs/bert_base_layer.yaml, the benchmark's default workload
        _case("linears_base_8x128", "linears", M=1024, D=768, F=3072),
        # configs/vit_base_model.yaml: 64 images of 197 tokens, a ragged last tile
        _case("linears_vit_64x197", "linears", M=64 * 197, D=768, F=3072),
        # a point of the hidden-size sweep: 256 codebooks whatever the width (v = 10), on 8 images
        _case("linears_h2560_8x197", "linears", M=8 * 197, D=2560, F=10240, v=10, scale=0.1, lut_bias=0.2),
        # a point of the centroid sweep: 64 sequences of 512 tokens, 64 centroids
        _case("linears_ct64_64x512", "linears", M=32768, D=768, F=3072, v=4, CT=64, scale=0.1, lut_bias=0.2),
        # configs/large_amm.yaml, the largest operator
        _case("amm_large_65536", "amm", M=65536, K=4096, N=16384),
        # the benchmark's end-to-end leg: the BERT-base linears with activations and results in host memory
        _case("host_base_8x128", "host", M=1024, D=768, F=3072),
        # a host that forbids allocation, one batch of 4 sequences through FFN1
        _case("static_ffn1_512", "static", M=512, K=768, N=3072),
        # converting a BERT-base FFN1 weight
        _case("build_ffn1", "build", K=768, N=3072),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# contraction steps of the largest listed case, and of the largest that the CUDA-core gather of `static` gets
_MOST = 65536 * 2048 * 16 * 16384
_MOST_STATIC = 8192 * 256 * 16 * 4096


def _steps(c):
    if c["kind"] == "build":
        return c["K"] * c["CT"] * c["N"]
    return sum(M * (K // v) * c["CT"] * N for M, K, N, v in _amms(c))


def draw(rng):
    """One more case: the kinds above at other token counts, widths, sub-vector lengths and centroid counts."""
    while True:
        kind = rng.choice(["amm", "amm", "linears", "linears", "layer", "host", "static", "build"])
        v, ct = rng.choice([(2, 8), (2, 16), (2, 32), (4, 8), (4, 16), (4, 32), (4, 64), (4, 128), (8, 8), (8, 16), (8, 32),
                            (10, 16), (16, 16), (20, 16), (32, 16)])
        c = _case("", kind, v=v, CT=ct)
        if rng.random() < 0.5:
            c.update(scale=0.1, lut_bias=0.2)   # the quantisation factors of the sweeps
        if kind in ("amm", "static", "build"):
            c.update(K=16 * v * _log_uniform(rng, max(1, 16 // v), 512 // v), N=16 * _log_uniform(rng, 12, 1024))   # 256..8192 -> 192..16384
            if kind != "build":
                c["M"] = _log_uniform(rng, 1, 65536 if kind == "amm" else 8192)
        else:
            D, heads = rng.choice([(768, 12), (1024, 16), (1280, 16), (2560, 32)])
            if D % (16 * v):
                continue
            c.update(D=D, F=4 * D)
            seq = _log_uniform(rng, 16, 512)
            batch = _log_uniform(rng, 1, 64 if kind == "linears" else 16)
            c.update(dict(batch=batch, seq=seq, heads=heads) if kind == "layer" else dict(M=batch * seq))
        if _steps(c) > (_MOST_STATIC if kind == "static" else _MOST):
            continue
        if kind == "static" and c["M"] * (c["K"] // v) > 8 << 20:   # LUTAMM_STATIC_SCRATCH_BYTES
            continue
        return c


def _amms(c):
    """(tokens, K, N, v) of each linear of the case."""
    if c["kind"] in ("amm", "static"):
        return [(c["M"], c["K"], c["N"], c["v"])]
    M = c["batch"] * c["seq"] if c["kind"] == "layer" else c["M"]
    D, F = c["D"], c["F"]
    return [(M, K, N, c["v"]) for K, N in ((D, 3 * D), (D, D), (D, F), (F, D))]


class _Session:
    """What a process keeps: one context on the GPU and the stream its calls are queued on."""
    _one = None

    def __init__(self):
        self.ctx = P.LutAmmContext(0)
        self.stream = torch.cuda.Stream()
        self.ctx.set_stream(self.stream.cuda_stream)
        self.ids = itertools.count(0, 8)

    @classmethod
    def get(cls):
        if cls._one is None:
            cls._one = cls()
        return cls._one


class _State:
    """Inputs, resident weights and output buffers of one case."""

    def __init__(self, case):
        self.case, self.s, self.loaded = case, _Session.get(), []

    def load(self, layer_id, weights):
        self.s.ctx.load_weights(layer_id, *weights)
        self.loaded.append(layer_id)

    def __del__(self):
        for lid in self.loaded:
            self.s.ctx.unload_weights(lid)


def _weights(gen, K, N, v, CT, scale, lut_bias):
    """Centroids N(0,1), table bytes uniform in [-127,127], bias N(0,0.02): the distributions of synth.py, on the GPU."""
    dev = dict(device="cuda", generator=gen)
    centroid = torch.randn(K // v, CT, v, **dev)
    lut = torch.randint(-127, 128, (K // v, CT, N), dtype=torch.int8, **dev)
    bias = torch.randn(N, **dev) * 0.02
    return centroid, lut, bias, scale, lut_bias


def prepare(case, seed):
    st = _State(case)
    with torch.cuda.stream(st.s.stream):
        gen = torch.Generator(device="cuda").manual_seed(seed)
        _fill(st, case, gen)
        st.s.stream.synchronize()
    return st


def _fill(st, case, gen):
    dev = dict(device="cuda", generator=gen)
    kind, v, CT = case["kind"], case["v"], case["CT"]
    if kind == "build":
        K, N = case["K"], case["N"]
        st.centroid = torch.randn(K // v, CT, v, **dev)
        st.weight = torch.randn(K, N, **dev) * 0.02
        st.lut = torch.empty(K // v, CT, N, dtype=torch.int8, device="cuda")
        return
    amms = _amms(case)
    weights = [_weights(gen, K, N, v, CT, case["scale"], case["lut_bias"]) for _, K, N, _ in amms]
    if kind == "layer":
        named = dict(zip(L.LINEARS, weights))
        ones, zeros = torch.ones(case["D"]).numpy(), torch.zeros(case["D"]).numpy()
        named.update(ln1=(ones, zeros), ln2=(ones, zeros))
        first = next(st.s.ids)
        st.layer = L.LutTransformerLayer(st.s.ctx, named, case["seq"], case["batch"], case["heads"], first_layer_id=first)
        st.loaded = list(st.layer.ids.values())
        st.x = torch.randn(amms[0][0], case["D"], **dev)
        return
    st.x = [torch.randn(M, K, **dev) for M, K, _, _ in amms]
    if kind == "static":
        (M, K, N, _), = amms
        st.w = weights[0]
        st.y = [torch.empty(M, N, device="cuda")]
        st.params = P.make_params(M, K, N, K // v, CT, case["scale"], case["lut_bias"])
        return
    first = next(st.s.ids)
    for k, w in enumerate(weights):
        st.load(first + k, w)
    st.y = [torch.empty(M, N, device="cuda") for M, _, N, _ in amms]
    if kind == "host":
        st.x = [x.cpu().pin_memory() for x in st.x]
        st.y = [torch.empty(y.shape, pin_memory=True) for y in st.y]


def run(state):
    kind, ctx = state.case["kind"], state.s.ctx
    if kind == "layer":
        with torch.cuda.stream(state.s.stream):
            return state.layer.forward(state.x)
    if kind == "build":
        return ctx.build_lut(state.centroid, state.weight, lut_out=state.lut)
    if kind == "static":
        centroid, lut, bias = state.w[:3]
        ip, lp = state.params
        lib = P.load_library()
        rc = lib.lutamm_amm_static_scratch(0, state.s.stream.cuda_stream, state.x[0].data_ptr(), centroid.data_ptr(), lut.data_ptr(),
                                           bias.data_ptr(), state.y[0].data_ptr(), ctypes.byref(ip), ctypes.byref(lp))
        if rc != P.OK:
            raise P.LutAmmError(rc, lib.lutamm_static_scratch_last_error().decode())
        return state.y
    for lid, x, y in zip(state.loaded, state.x, state.y):
        ctx.amm_host(lid, x, y, flags=P.FLAG_ASYNC)
    if kind == "host":
        ctx.sync()
    return state.y


def work(case):
    """Activations, centroids, table and bias read once, results written once; three operations per centroid
    component of the search, one addition per table byte a token selects, three per output."""
    if case["kind"] == "build":
        K, N, CT, v = case["K"], case["N"], case["CT"], case["v"]
        return {"bytes": 4 * K * N + 4 * K * CT + (K // v) * CT * N, "flops": 2 * K * CT * N}
    nbytes = flops = 0
    for M, K, N, v in _amms(case):
        CB, CT = K // v, case["CT"]
        nbytes += 4 * M * K + 4 * K * CT + CB * CT * N + 4 * N + 4 * M * N
        flops += 3 * M * K * CT + M * CB * N + 3 * M * N
    if case["kind"] == "layer":   # the two attention products
        B, S, D = case["batch"], case["seq"], case["D"]
        flops += 4 * B * S * S * D
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    return "exact"
