"""Split-K of the tiled dense kernel (a tile's K blocks over a cluster, partial tiles added through
distributed shared memory) against the same tiles without it."""
import pytest
import torch

from oracle import blockscale_ref as O
from tests.test_plans import DECODE, TILED, _gemm_plan

pytestmark = pytest.mark.gpu


def _bound(ref, a, b, extra):
    """One rounding of the fp16 result (2^-10 covers an ulp) and, for sums in another order, 2^-24 per
    addition (K blocks + CTAs) of the sum of the products' magnitudes."""
    return 2.0 ** -10 * ref.abs() + 2.0 ** -24 * extra * (a.abs() @ b.abs().t()) + 2.0 ** -24


# M: fewer rows than CTAs, one row in the last row block, slices of unequal length; N: a multiple of 16
# only, fewer columns than a tile; K: one K block per CTA, a shorter last range. Every cluster size the
# automatic plan may choose, where each of its CTAs has K blocks.
SHAPES = [(1, 512, 512), (7, 528, 1152), (129, 528, 896), (129, 528, 2048), (300, 1040, 1152), (255, 256, 8320)]


def _splits(K, most):
    blocks = K // 128
    each = {s: -(-blocks // s) for s in range(2, most + 1)}
    return [s for s in each if -(-blocks // each[s]) == s]


@pytest.mark.parametrize("M,N,K,block_n,split_k", [(M, N, K, bn, s) for M, N, K in SHAPES for bn in (64, 128, 256)
                                                   for s in _splits(K, 4 if bn == 256 else 8)])
def test_split_k_matches_unsplit(M, N, K, block_n, split_k):
    from flydsl_b200 import _lib
    from flydsl_b200.kernels import compile_blockscale_preshuffle_gemm
    from flydsl_b200.utils import shuffle_weight

    assert _gemm_plan(M, N, K, sms=0, block_n=block_n, path=TILED, split_k=split_k)["splits"] == split_k
    case = O.make_dense_case(M, N, K, seed=M + N + K)
    b = shuffle_weight(case["b_q"].cuda())
    sa, sb = case["a_scale"].cuda().t().contiguous(), case["b_scale"].cuda().contiguous()
    out = []
    for sp in (1, split_k, split_k):
        fn = compile_blockscale_preshuffle_gemm(M=M, N=N, K=K, tile_m=64, tile_n=128, tile_k=128, out_dtype="fp16",
                                                block_n=block_n, path="tiled", split_k=sp)
        c = torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
        fn(c, case["a_q"].cuda(), b, sa, sb, M, N, None)
        assert _lib.query_device_error() == 0
        out.append(c.float())
    a = (case["a_q"].cuda().float().view(M, -1, 128) * case["a_scale"].cuda().unsqueeze(-1)).view(M, K)
    w = case["b_q"].cuda().float() * O.expand_weight_scale(case["b_scale"].cuda(), N, K)
    assert ((out[1] - out[0]).abs() <= _bound(out[0], a, w, K // 128 + split_k)).all()
    assert torch.equal(out[1], out[2])   # rank order: the same bits every time


@pytest.mark.parametrize("M,N,K", [(65, 256, 4096), (129, 1040, 7168), (777, 1536, 7168), (1000, 528, 8320)])
def test_split_k_pertoken(M, N, K):
    """The automatic choice splits these; path="tiled" does not."""
    from flydsl_b200 import _lib
    from flydsl_b200.kernels import compile_preshuffle_gemm_a8
    from flydsl_b200.utils import quant_pertoken, shuffle_weight

    assert _gemm_plan(M, N, K, pertoken=True, sms=0)["splits"] > 1
    assert _gemm_plan(M, N, K, pertoken=True, sms=0, path=TILED)["splits"] == 1
    g = torch.Generator("cuda").manual_seed(M + N)
    a_q, sa = quant_pertoken(torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16))
    w = torch.randn(N, K, generator=g, device="cuda").to(torch.float8_e4m3fn)
    sb = torch.rand(N, generator=g, device="cuda") + 0.5
    out = []
    for path in ("tiled", "auto", "auto"):
        fn = compile_preshuffle_gemm_a8(M=M, N=N, K=K, tile_m=64, tile_n=128, tile_k=128, out_dtype="fp16", path=path)
        c = torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
        fn(c, a_q, shuffle_weight(w), sa, sb, M, N, None)
        assert _lib.query_device_error() == 0
        out.append(c.float())
    bound = _bound(out[0], a_q.float() * sa.view(M, 1), w.float() * sb.view(N, 1), K // 32 + 4)
    assert ((out[1] - out[0]).abs() <= bound).all()
    assert torch.equal(out[1], out[2])


# Decode-size M on both sides of the choice between the decode and the tiled kernel
@pytest.mark.parametrize("M,N,K,kernel", [(1, 528, 1536, DECODE), (1, 2064, 3072, DECODE), (1, 7056, 7168, TILED),
                                          (8, 2064, 2048, DECODE), (8, 12288, 5120, TILED), (16, 1552, 2048, DECODE),
                                          (16, 12688, 1920, TILED), (17, 1040, 3072, DECODE), (17, 1552, 2560, DECODE),
                                          (17, 7040, 512, TILED), (32, 2192, 2048, TILED), (32, 7168, 4224, TILED),
                                          (24, 9600, 2304, TILED), (33, 1536, 2048, TILED), (33, 12160, 4096, TILED)])
def test_decode_or_tiled(M, N, K, kernel):
    from flydsl_b200 import _lib
    from flydsl_b200.kernels import compile_blockscale_preshuffle_gemm
    from flydsl_b200.utils import shuffle_weight

    assert _gemm_plan(M, N, K, sms=0)["kernel"] == kernel
    case = O.make_dense_case(M, N, K, seed=M + N)
    b = shuffle_weight(case["b_q"].cuda())
    sa, sb = case["a_scale"].cuda().t().contiguous(), case["b_scale"].cuda().contiguous()
    out = []
    for path in ("auto", "tiled"):
        fn = compile_blockscale_preshuffle_gemm(M=M, N=N, K=K, tile_m=64, tile_n=128, tile_k=128, out_dtype="fp16", path=path)
        c = torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
        fn(c, case["a_q"].cuda(), b, sa, sb, M, N, None)
        assert _lib.query_device_error() == 0
        out.append(c.float())
    a = (case["a_q"].cuda().float().view(M, -1, 128) * case["a_scale"].cuda().unsqueeze(-1)).view(M, K)
    w = case["b_q"].cuda().float() * O.expand_weight_scale(case["b_scale"].cuda(), N, K)
    assert ((out[0] - out[1]).abs() <= _bound(out[1], a, w, K // 128 + 8)).all()
