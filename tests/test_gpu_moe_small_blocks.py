"""MoE stages with the weights on the MMA's M side (routing blocks of at most 32 rows) against the tiled
kernel on the same inputs: exact fp8 products, the same order of fp32 additions, so the same bits."""
import pytest
import torch

from oracle import blockscale_ref as O

pytestmark = pytest.mark.gpu


# block sizes of every accumulator width, merged neighbours (hot experts: runs of an odd and an even
# number of blocks), one token, model_dim with an odd number of 128-channel tiles, one K block, experts
# without tokens
SHAPES = [(1, 256, 128, 4, 1, 16), (7, 512, 256, 8, 2, 8), (96, 1024, 512, 16, 4, 32), (33, 640, 384, 8, 3, 24),
          (200, 1152, 640, 6, 2, 32), (70, 1152, 256, 4, 3, 16)]


def _case(T, H, I, E, k):
    m = O.make_moe_case(T=T, H=H, I=I, E=E, topk=k, seed=T + H, hot_experts=1, hot_bias=2.0)
    return {a: v.cuda() if torch.is_tensor(v) else v for a, v in m.items()}


@pytest.mark.parametrize("T,H,I,E,k,tile_m", SHAPES)
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float16])
def test_block_scale_layer(T, H, I, E, k, tile_m, out_dtype):
    from flydsl_b200 import _lib
    from flydsl_b200.moe import BlockscaleMoE

    m = _case(T, H, I, E, k)
    args = (m["x_q"], m["x_scale"].t().contiguous(), m["topk_ids"], m["topk_weights"])
    out = {}
    for mode in ("reduce", "atomic"):
        for layout in (False, True, None):   # gathered, routing order, the layer's choice
            layer = BlockscaleMoE.from_unpacked(m["w1_q"], m["w1_scale"], m["w2_q"], m["w2_scale"], topk=k, tile_m=tile_m,
                                                mode=mode, sorted_layout=layout, out_dtype=out_dtype)
            out[mode, layout] = layer.forward(*args).float()
            assert _lib.query_device_error() == 0
    assert torch.equal(out["reduce", True], out["reduce", False])
    assert torch.equal(out["reduce", None], out["reduce", False])
    # 16-bit atomics round the running sum at each of the k additions, in any order: k half ulps of the
    # largest partial sum, which 4 times the largest result covers for these weights (softmax, sum 1)
    ulp = 2.0 ** -8 if out_dtype == torch.bfloat16 else 2.0 ** -11
    scale = out["reduce", True].abs().max()
    for layout in (True, None):
        assert (out["atomic", layout] - out["reduce", True]).abs().max() <= (k + 1) * ulp * 4 * scale


@pytest.mark.parametrize("T,H,I,E,k,tile_m", SHAPES)
def test_pertoken_layer(T, H, I, E, k, tile_m):
    from flydsl_b200 import _lib
    from flydsl_b200.moe import PertokenMoE
    from flydsl_b200.utils import quant_pertoken, shuffle_weight

    m = _case(T, H, I, E, k)
    g = torch.Generator("cuda").manual_seed(T)
    w1 = shuffle_weight(torch.randn(E, 2 * I, H, device="cuda", generator=g).to(torch.float8_e4m3fn))
    w2 = shuffle_weight(torch.randn(E, H, I, device="cuda", generator=g).to(torch.float8_e4m3fn))
    s1 = torch.rand(E, 2 * I, device="cuda", generator=g) * 0.02 + 0.01
    s2 = torch.rand(E, H, device="cuda", generator=g) * 0.02 + 0.01
    x_q, x_s = quant_pertoken(torch.randn(T, H, device="cuda", generator=g).to(torch.bfloat16))
    out = []
    for t in (tile_m, 128):
        layer = PertokenMoE(w1, s1, w2, s2, topk=k, tile_m=t)
        out.append(layer.forward(x_q, x_s, m["topk_ids"], m["topk_weights"]))
        assert _lib.query_device_error() == 0
    assert torch.equal(*out)


def test_more_blocks_than_the_list_and_blocks_without_expert():
    """Routing arrays a caller may bring: blocks marked -1 between those of an expert, and more blocks
    than the kernel's list of token tiles holds (no merging then)."""
    from flydsl_b200 import _lib
    from flydsl_b200.kernels.moe_blockscale_2stage import compile_moe_blockscale_gemm1

    T, H, I, E, k, tile_m = 33000, 256, 128, 4, 1, 8
    m = _case(T, H, I, E, k)
    from flydsl_b200.utils import moe_gather_rows, shuffle_weight

    L = T * k + E * tile_m - k
    for blocks in (4110, 301):
        ids = torch.full((L,), (k << 24) | T, dtype=torch.int32, device="cuda")
        n = blocks * tile_m   # one token in each block
        ids[:n:tile_m] = torch.arange(blocks, dtype=torch.int32, device="cuda")
        eid = (torch.arange(L // tile_m + 1, dtype=torch.int32, device="cuda") // 3) % E
        eid[5::7] = -1
        npp = torch.tensor([n, T], dtype=torch.int32, device="cuda")
        x, xs = moe_gather_rows(m["x_q"], m["x_scale"].t().contiguous(), ids, npp, topk=k)
        w = shuffle_weight(m["w1_q"])
        out = []
        for block_n in (None, 256):   # a tile width asks for the tiled kernel
            fn = compile_moe_blockscale_gemm1(model_dim=H, inter_dim=I, experts=E, topk=k, tile_m=tile_m, tile_n=256,
                                              tile_k=128, doweight_stage1=False, out_dtype="f16", a_sorted=True,
                                              out_sorted=True, block_n=block_n)
            o = torch.zeros((L, I), dtype=torch.float16, device="cuda")
            fn(o, x, w, xs, m["w1_scale"].contiguous(), ids, eid, torch.ones(L, device="cuda"), npp, T, I, H, blocks, None)
            assert _lib.query_device_error() == 0
            out.append(o)
        assert torch.equal(*out)
        assert out[0].abs().sum() > 0


@pytest.mark.parametrize("tokens,rows", [(80, 66), (66, 80)])
def test_routing_of_another_number_of_tokens(tokens, rows):
    """Fewer routed tokens than activation rows (the others get nothing), or more (dropped): layers with
    small blocks take these as the layers with gathered activations do."""
    from flydsl_b200 import _lib
    from flydsl_b200.moe import BlockscaleMoE

    H, I, E, k = 512, 256, 8, 2
    m = _case(80, H, I, E, k)
    args = (m["x_q"][:tokens], m["x_scale"][:tokens].t().contiguous(), m["topk_ids"][:rows], m["topk_weights"][:rows])
    both = min(tokens, rows)
    for mode in ("reduce", "atomic"):
        out = []
        for layout in (None, False):
            layer = BlockscaleMoE.from_unpacked(m["w1_q"], m["w1_scale"], m["w2_q"], m["w2_scale"], topk=k, tile_m=16,
                                                mode=mode, sorted_layout=layout)
            assert layer._small_pays_off(tokens)
            out.append(layer.forward(*args))
            assert _lib.query_device_error() == 0 and out[-1].shape == (tokens, H)
        if mode == "reduce":   # rows without routes are unspecified there
            assert torch.equal(out[0][:both], out[1][:both])
        else:
            assert not out[0][both:].any() and not out[1][both:].any()
            scale = out[1].float().abs().max()
            assert (out[0].float() - out[1].float()).abs().max() <= (k + 1) * 2.0 ** -8 * 4 * scale
