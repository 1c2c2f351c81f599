"""The workloads by which this framework's speed is measured: what a serving program has it do,
through the public launchers and layers, from the smallest decode call to the largest prefill.

Five kinds of work:

``dense``     FP8 block-scale GEMM (``compile_blockscale_preshuffle_gemm``); with ``quantise`` the
              call starts from bf16 activations (``quant_1x128``), as a linear layer does
``pertoken``  its sibling with one scale per token and per output channel
              (``compile_preshuffle_gemm_a8``); ``quantise`` as above (``quant_pertoken``)
``int4``      weight-only int4 x bf16 GEMM (``compile_int4_weight_only_gemm``)
``moe``       the two-stage block-scale MoE: router logits -> top-k -> activations quantised ->
              routing sort, both stages, combine (``route_topk``, ``quant_1x128``, ``BlockscaleMoE``)
``ptmoe``     the same with per-token scales (``quant_pertoken``, ``PertokenMoE``)

Sizes are those of the benchmark (the three (N, K) pairs, M from 1 to 16384, the 256-expert top-8
layer with 7168 x 2048 experts at 32 to 4096 tokens, skewed routing with 16 hot experts) and of the
reference's test grids, with ragged ones among them. Weights are N(0, 0.02), activations and router
logits N(0, 1), quantised with scale = amax / 448 per group (int4: amax / 7).
"""
import math

import torch

from flydsl_b200.kernels import (
    compile_blockscale_preshuffle_gemm,
    compile_int4_weight_only_gemm,
    compile_preshuffle_gemm_a8,
    pack_int4_weight,
)
from flydsl_b200.moe import BlockscaleMoE, PertokenMoE
from flydsl_b200.utils import quant_1x128, quant_pertoken, route_topk, shuffle_weight

FP8 = torch.float8_e4m3fn
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def listed():
    return [
        # one sequence decoding: the smallest call, all latency
        {"name": "dense_m1", "kind": "dense", "M": 1, "N": 7168, "K": 2048, "out": "bf16", "quantise": False},
        # a decode batch through a wide (fused q/k/v or up) projection, from bf16 activations
        {"name": "dense_m32_wide", "kind": "dense", "M": 32, "N": 24576, "K": 1536, "out": "bf16", "quantise": True},
        # a short chunk of prefill through a deep down projection
        {"name": "dense_m256_deep", "kind": "dense", "M": 256, "N": 4096, "K": 7168, "out": "bf16",
         "quantise": False},
        # a ragged chunk through the narrow low-rank projection, fp16 outputs, from activations
        {"name": "dense_m777_narrow", "kind": "dense", "M": 777, "N": 1536, "K": 7168, "out": "fp16",
         "quantise": True},
        # the benchmark's headline GEMM
        {"name": "dense_m4096", "kind": "dense", "M": 4096, "N": 7168, "K": 2048, "out": "bf16", "quantise": False},
        # the largest prefill batch of the sweep
        {"name": "dense_m16384_deep", "kind": "dense", "M": 16384, "N": 4096, "K": 7168, "out": "bf16",
         "quantise": False},
        # per-token scales, the large shape of the reference's test grid
        {"name": "pertoken_m5120", "kind": "pertoken", "M": 5120, "N": 5120, "K": 8320, "out": "fp16",
         "quantise": False},
        # int4 weights, a decode batch
        {"name": "int4_m16", "kind": "int4", "M": 16, "N": 8192, "K": 8192},
        # MoE decode, few tokens, some experts hot: most experts see no token or one
        {"name": "moe_t32_skewed", "kind": "moe", "T": 32, "H": 7168, "I": 2048, "E": 256, "topk": 8, "hot": 16,
         "mode": "reduce"},
        # MoE decode at a full batch
        {"name": "moe_t256_skewed", "kind": "moe", "T": 256, "H": 7168, "I": 2048, "E": 256, "topk": 8, "hot": 16,
         "mode": "reduce"},
        # MoE prefill: the benchmark's layer
        {"name": "moe_t4096", "kind": "moe", "T": 4096, "H": 7168, "I": 2048, "E": 256, "topk": 8, "hot": 0,
         "mode": "reduce"},
        # per-token-scale MoE on a ragged batch
        {"name": "ptmoe_t1000", "kind": "ptmoe", "T": 1000, "H": 7168, "I": 2048, "E": 256, "topk": 8, "hot": 0},
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of ``step`` in [lo, hi], spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(hi, max(lo, step * round(v / step))))


def draw(rng):
    kind = rng.choices(["dense", "pertoken", "int4", "moe", "ptmoe"], [40, 15, 15, 20, 10])[0]
    if kind == "int4":
        return {"kind": kind, "M": _log(rng, 1, 64), "N": _log(rng, 1024, 16384, 128), "K": _log(rng, 1024, 8192, 128)}
    if kind in ("dense", "pertoken"):
        # N is a multiple of 128 for most weights; 16 is what the layout asks for
        step = 128 if rng.random() < 0.7 else 16
        case = {"kind": kind, "M": _log(rng, 1, 16384),
                "N": _log(rng, 1024, 8192 if rng.random() < 0.7 else 24576, step),
                "K": _log(rng, 1024, 8320, 128), "out": rng.choice(["bf16", "bf16", "fp16"]),
                "quantise": rng.random() < 0.4}
        case["M"] = min(case["M"], 10**12 // (case["N"] * case["K"]))
        return case
    E = rng.choice([32, 64, 128, 256])
    case = {"kind": kind, "T": _log(rng, 4, 4096), "H": _log(rng, 1024, 7168, 128), "I": _log(rng, 256, 2048, 128),
            "E": E, "topk": rng.choice([2, 4, 6, 8]), "hot": rng.choice([0, 0, E // 16])}
    if kind == "moe":
        case["mode"] = rng.choice(["reduce", "reduce", "atomic"])
    return case


def _tile_m(tokens):
    """Routing block size by batch, as the benchmark chooses it."""
    return 128 if tokens >= 1024 else 32 if tokens >= 256 else 16


def _block_quant(w):
    """128x128 amax blocks: fp8 ``[N, K]`` and scales ``[ceil(N/128), K/128]``."""
    n, k = w.shape
    pad = -n % 128
    g = torch.nn.functional.pad(w, (0, 0, 0, pad)).view((n + pad) // 128, 128, k // 128, 128)
    s = g.abs().amax(dim=(1, 3), keepdim=True) / 448.0
    s[s == 0] = 1
    return (g / s).to(FP8).view(n + pad, k)[:n], s.view((n + pad) // 128, k // 128)


def _channel_quant(w):
    """One amax scale per output channel: fp8 ``[N, K]`` and scales ``[N]``."""
    s = w.abs().amax(dim=1, keepdim=True) / 448.0
    s[s == 0] = 1
    return (w / s).to(FP8), s.view(-1)


def _experts(E, n, k, quant, gen):
    """Weights of E experts, quantised one by one: fp8 ``[E, n, k]`` and scales ``[E, -1]``."""
    q, scales = torch.empty((E, n, k), dtype=FP8, device="cuda"), []
    w = torch.empty((n, k), device="cuda")
    for e in range(E):
        q[e], s = quant(w.normal_(0.0, 0.02, generator=gen))
        scales.append(s.reshape(-1))
    return q, torch.stack(scales)


def _inputs(case, seed):
    """Activations, quantised weights in row-major order and router logits, from the seed alone."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    d = {}

    def normal(*shape):
        return torch.randn(*shape, generator=gen, device="cuda")

    if kind in ("dense", "pertoken"):
        M, N, K = case["M"], case["N"], case["K"]
        w = normal(N, K) * 0.02
        d["x"] = normal(M, K).to(torch.bfloat16)
        d["w"], d["w_scale"] = (_block_quant if kind == "dense" else _channel_quant)(w)
        return d
    if kind == "int4":
        M, N, K = case["M"], case["N"], case["K"]
        g = (normal(N, K) * 0.02).view(N, K // 128, 128)
        s = (g.abs().amax(dim=-1) / 7.0).to(torch.bfloat16)
        s[s == 0] = 1
        d["w"] = torch.round(g / s.float().unsqueeze(-1)).clamp_(-8, 7).to(torch.int8).view(N, K)
        d["w_scale"] = s
        d["x"] = normal(M, K).to(torch.bfloat16)
        return d
    T, H, I, E = case["T"], case["H"], case["I"], case["E"]
    quant = _block_quant if kind == "moe" else _channel_quant
    d["w1"], d["w1_scale"] = _experts(E, 2 * I, H, quant, gen)
    d["w2"], d["w2_scale"] = _experts(E, H, I, quant, gen)
    d["x"] = normal(T, H).to(torch.bfloat16)
    d["logits"] = normal(T, E)
    d["logits"][:, :case["hot"]] += 2.0
    return d


def prepare(case, seed):
    kind = case["kind"]
    d = _inputs(case, seed)
    state = {**case, **d}
    if kind in ("dense", "pertoken"):
        M, N, K = case["M"], case["N"], case["K"]
        shape = dict(M=M, N=N, K=K, tile_m=64, tile_n=128, tile_k=128, out_dtype=case["out"])
        compile_gemm = compile_blockscale_preshuffle_gemm if kind == "dense" else compile_preshuffle_gemm_a8
        state["gemm"] = compile_gemm(**shape)
        state["w"] = shuffle_weight(d["w"].contiguous())
        state["c"] = torch.empty((M, N), dtype=DTYPES[case["out"]], device="cuda")
        if not case["quantise"]:
            state["x_q"], state["x_scale"] = (quant_1x128 if kind == "dense" else quant_pertoken)(state.pop("x"))
        return state
    if kind == "int4":
        M, N, K = case["M"], case["N"], case["K"]
        state["w"], state["w_scale"] = pack_int4_weight(d["w"], d["w_scale"])
        state["gemm"] = compile_int4_weight_only_gemm(N=N, K=K)
        state["c"] = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
        return state
    for name in ("w1", "w2"):
        d[name] = None
        state[name] = shuffle_weight(state[name])
    weights = [state.pop(name) for name in ("w1", "w1_scale", "w2", "w2_scale")]
    if kind == "moe":
        state["layer"] = BlockscaleMoE(*weights, topk=case["topk"], tile_m=_tile_m(case["T"]), mode=case["mode"])
    else:
        state["layer"] = PertokenMoE(*weights, topk=case["topk"], tile_m=_tile_m(case["T"]))
    state["out"] = torch.empty((case["T"], case["H"]), dtype=torch.bfloat16, device="cuda")
    return state


def run(state):
    kind = state["kind"]
    if kind in ("dense", "pertoken"):
        if state["quantise"]:
            x_q, x_scale = (quant_1x128 if kind == "dense" else quant_pertoken)(state["x"])
        else:
            x_q, x_scale = state["x_q"], state["x_scale"]
        state["gemm"](state["c"], x_q, state["w"], x_scale, state["w_scale"], state["M"], state["N"], None)
        return state["c"]
    if kind == "int4":
        state["gemm"](state["c"], state["x"], state["w"], state["w_scale"], state["M"], None)
        return state["c"]
    ids, weights = route_topk(state["logits"], state["topk"])
    x_q, x_scale = (quant_1x128 if kind == "moe" else quant_pertoken)(state["x"])
    return state["layer"].forward(x_q, x_scale, ids, weights, out=state["out"])


def _above(z):
    """Probability of a standard normal value above z."""
    return 0.5 * math.erfc(z / math.sqrt(2.0))


def work(case):
    """Each input read once, each output written once; a MoE reads the weights of the experts that
    receive tokens (their expected number), and its intermediates stay on the chip."""
    kind = case["kind"]
    if kind in ("dense", "pertoken"):
        M, N, K = case["M"], case["N"], case["K"]
        x = 2 * M * K if case["quantise"] else M * K + 4 * M * (K // 128 if kind == "dense" else 1)
        scales = 4 * ((N + 127) // 128) * (K // 128) if kind == "dense" else 4 * N
        return {"bytes": x + N * K + scales + 2 * M * N, "flops": 2 * M * N * K}
    if kind == "int4":
        M, N, K = case["M"], case["N"], case["K"]
        return {"bytes": N * K // 2 + 2 * N * (K // 128) + 2 * M * K + 2 * M * N, "flops": 2 * M * N * K}
    T, H, I, E, k = case["T"], case["H"], case["I"], case["E"], case["topk"]
    # chance of a hot (logit raised by 2) and of another expert to be among a token's top k: both are
    # above the threshold that k experts exceed on average
    hot, lo, hi = case["hot"], -6.0, 8.0
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if hot * _above(mid - 2.0) + (E - hot) * _above(mid) > k else (lo, mid)
    active = hot * (1 - (1 - _above(lo - 2.0)) ** T) + (E - hot) * (1 - (1 - _above(lo)) ** T)
    scales = 4 * (3 * H * I // (128 * 128)) if kind == "moe" else 4 * (2 * I + H)
    return {"bytes": active * (3 * H * I + scales) + 2 * T * H + 4 * T * E + 2 * T * H,
            "flops": 2 * T * k * 3 * H * I}


def tolerance(case):
    """About four times what the results differ from the same computation in 64 bits: rounding of the
    16-bit output alone for the GEMMs (bf16 1.7e-3, largest 3.9e-3; fp16 2.1e-4, 4.9e-4); for the layers
    also the fp8 rounding of the intermediate, where a difference in the last bit of a stage-1 value
    can flip a code (2.8e-3, 4.4e-2), and with atomic adds one bf16 rounding per expert."""
    if case["kind"] in ("moe", "ptmoe"):
        return {"rel": 2e-2, "max": 0.2} if case.get("mode") == "atomic" else {"rel": 1e-2, "max": 0.17}
    return {"rel": 8.5e-4, "max": 2e-3} if case.get("out") == "fp16" else {"rel": 6.6e-3, "max": 1.6e-2}


def _quantised(x, group, dtype=torch.float64):
    """The values, in 64 bits, that rows quantised in groups of ``group`` stand for; scale and code
    are computed in ``dtype``, by division (torch multiplies by the reciprocal of a Python number,
    which moves values that lie halfway between two codes)."""
    g = x.to(dtype).view(x.shape[0], -1, group)
    s = g.abs().amax(dim=-1, keepdim=True)
    s = s / torch.full_like(s, 448.0)
    s[s == 0] = 1
    return ((g / s).to(FP8).double() * s.double()).view(x.shape)


def _weight(w, scale, kind):
    """The values, in 64 bits, that one quantised weight ``[N, K]`` stands for."""
    n, k = w.shape
    if kind in ("pertoken", "ptmoe"):
        return w.double() * scale.double().view(n, 1)
    s = scale.double().view(-1, k // 128).repeat_interleave(128, dim=0)[:n]
    return (w.double().view(n, -1, 128) * s.unsqueeze(-1)).view(n, k)


def exact(case, seed):
    """``run``'s results by dequantised products in 64 bits. What a layer's formats define stays: the
    fp8 codes and 32-bit scales of its activations, and the fp8 grid of its intermediate."""
    kind = case["kind"]
    d = _inputs(case, seed)
    x = d["x"]
    if kind == "int4":
        n, k = d["w"].shape
        w = (d["w"].double().view(n, -1, 128) * d["w_scale"].double().unsqueeze(-1)).view(n, k)
        return x.double() @ w.t()
    x = _quantised(x, 128 if kind in ("dense", "moe") else x.shape[1], torch.float32)
    if kind in ("dense", "pertoken"):
        return x @ _weight(d["w"], d["w_scale"], kind).t()
    I = case["I"]
    values, ids = torch.topk(d["logits"], case["topk"], dim=-1)
    weights = torch.softmax(values.double(), dim=-1)
    out = torch.zeros_like(x)
    for e in range(case["E"]):
        token, slot = (ids == e).nonzero(as_tuple=True)
        if token.numel() == 0:
            continue
        y = x[token] @ _weight(d["w1"][e], d["w1_scale"][e], kind).t()
        act = _quantised(torch.nn.functional.silu(y[:, :I]) * y[:, I:], 128 if kind == "moe" else I)
        y = act @ _weight(d["w2"][e], d["w2_scale"][e], kind).t()
        out.index_add_(0, token, y * weights[token, slot].unsqueeze(-1))
    return out
