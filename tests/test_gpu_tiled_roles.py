"""Tiled block-scale kernel: the hand-overs between copier, issuer and epilogue warps (kept as counters) at the
edges of the ring, of the accumulator buffers and of the scale ring, against the oracle; several tiles per CTA."""
import pytest
import torch

from oracle import blockscale_ref as O
from tests.helpers import assert_close_to_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block_n", [32, 64, 128, 256])
@pytest.mark.parametrize("M,N,K,max_ctas", [
    (17, 272, 128, 0), (40, 144, 256, 1),    # one and two K blocks: fewer than stages, buffers or scale slots
    (129, 528, 1152, 1),                     # one CTA walks every tile: counters run on from tile to tile
    (300, 304, 1408, 3), (64, 256, 2560, 1), # eleven and twenty K blocks: rings of 3 to 10 stages wrap unevenly
])
def test_tiled_counters(M, N, K, max_ctas, block_n):
    from flydsl_b200 import _lib
    from flydsl_b200.kernels import compile_blockscale_preshuffle_gemm
    from flydsl_b200.utils import shuffle_weight

    c = O.make_dense_case(M, N, K, seed=M + N + K)
    ref = O.run_torch_blockscale(c["a_q"], c["b_q"], c["a_scale"], c["b_scale"], dtype=torch.float32)
    fn = compile_blockscale_preshuffle_gemm(M=M, N=N, K=K, tile_m=64, tile_n=128, tile_k=128, path="tiled",
                                            block_n=block_n)
    fn._cfg.max_ctas = max_ctas
    out = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    fn(out, c["a_q"].cuda(), shuffle_weight(c["b_q"].cuda()), c["a_scale"].cuda().t().contiguous(), c["b_scale"].cuda(),
       M, N, None)
    assert _lib.query_device_error() == 0
    assert_close_to_oracle(out, ref, f"tiled {M} {N} {K} bn={block_n} ctas={max_ctas}")


@pytest.mark.parametrize("M,N,K", [(1, 4096, 1024), (8, 7168, 2048), (16, 2688, 1408), (16, 8192, 5120), (17, 6912, 2560),
                                   (32, 2192, 1920), (32, 2560, 4992), (33, 7168, 7168), (64, 10240, 3968),
                                   (64, 1040, 7168)])
def test_decode_sizes_on_the_tiled_kernel_equal_the_decode_kernel(M, N, K):
    """Both edges of each token range of the dispatch rule; the two kernels differ in the order of sums over K."""
    from flydsl_b200 import _lib
    from flydsl_b200.kernels import compile_blockscale_preshuffle_gemm
    from tests.test_plans import TILED, _gemm_plan

    assert _gemm_plan(M, N, K, sms=0)["kernel"] == TILED
    gen = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, generator=gen, device="cuda").to(torch.float8_e4m3fn)
    b = torch.randn(N, K, generator=gen, device="cuda").to(torch.float8_e4m3fn)
    sa = torch.rand(K // 128, M, generator=gen, device="cuda") + 0.5
    sb = torch.rand((N + 127) // 128, K // 128, generator=gen, device="cuda") + 0.5
    outs = []
    for path in ("auto", "decode"):
        fn = compile_blockscale_preshuffle_gemm(M=M, N=N, K=K, tile_m=64, tile_n=128, tile_k=128, path=path)
        outs.append(torch.empty((M, N), dtype=torch.bfloat16, device="cuda"))
        fn(outs[-1], a, b, sa, sb, M, N, None)
    assert _lib.query_device_error() == 0
    # one rounding to bf16 (2^-8 of a value) on either side, sums in another order below it
    assert_close_to_oracle(outs[0], outs[1].float().cpu(), f"decode size {M} {N} {K}")
