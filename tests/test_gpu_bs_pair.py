"""Block-scale GEMM on CTA pairs (bs_pair_gemm.cu): which calls take it, and that it gives bit for bit what
the tiled kernel gives (same products, same order of sums)."""
import ctypes

import pytest
import torch

from flydsl_b200 import _lib

TILED, DECODE, PAIR = 1, 2, 3


def _plan(M, N, K, sms=148, **cfg):
    cfg = _lib.GemmCfg(*[cfg.get(name, 0) for name in ("block_n", "max_ctas", "path", "split_k")])
    plan = (ctypes.c_int32 * 5)()
    _lib.check(_lib.load().flyb200_gemm_plan(0, M, N, K, ctypes.byref(cfg), sms, plan))
    return dict(zip(("kernel", "block_n", "splits", "kbps", "ctas"), plan))


def test_pairs_only_where_the_tiled_kernel_would_run_unsplit_in_wide_tiles():
    seen = 0
    for M in (1, 64, 65, 128, 129, 256, 257, 313, 512, 777, 1093, 1126, 4096, 5000, 16384):
        for N in (16, 128, 1536, 3328, 4112, 7168, 12000, 24576):
            for K in (128, 1024, 2048, 7168):
                plan, tiled = _plan(M, N, K), _plan(M, N, K, path=TILED)
                if plan["kernel"] != PAIR:
                    continue
                seen += 1
                pairs = -(-M // 256) * -(-N // 256)
                assert plan["ctas"] == 2 * min(74, pairs) and plan["splits"] == 1 and tiled["block_n"] == 256
                # never more rounds than the tiled kernel needs, rarely more padding
                assert -(-pairs // 74) <= -(-(-(-M // 128) * -(-N // 256)) // 148)
                assert M >= 512 or -(-M // 128) % 2 == 0
                for asked in (dict(path=TILED), dict(block_n=256), dict(split_k=1), dict(max_ctas=1)):
                    assert _plan(M, N, K, **asked)["kernel"] != PAIR
                assert _plan(M, N, K, max_ctas=20)["ctas"] <= 20
    assert seen > 50


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,out,max_ctas", [
    (256, 256, 128, "bf16", 2),        # one tile, one K block
    (129, 128, 384, "bf16", 2),        # second column half and most of the second CTA's rows are padding
    (200, 144, 640, "fp16", 2),        # 16 columns in the second half
    (400, 272, 896, "bf16", 2),        # remainders in M and N, several tiles a pair, K blocks not a multiple of 4
    (777, 1552, 1152, "fp16", 6),
    (2500, 400, 256, "bf16", 4),       # fewer K blocks than stages and scale slots
    (4096, 7168, 2048, "bf16", 0),     # whole GPU, a ragged last round
    (9000, 1024, 7168, "bf16", 0),     # row blocks in groups, the last one short
])
def test_pairs_equal_the_tiled_kernel(M, N, K, out, max_ctas):
    from flydsl_b200.kernels import compile_blockscale_preshuffle_gemm

    gen = torch.Generator(device="cuda").manual_seed(M + N + K)
    dtype = {"bf16": torch.bfloat16, "fp16": torch.float16}[out]
    a = torch.randn(M, K, generator=gen, device="cuda").to(torch.float8_e4m3fn)
    b = torch.randn(N, K, generator=gen, device="cuda").to(torch.float8_e4m3fn)
    sa = torch.rand(K // 128, M, generator=gen, device="cuda") * 0.02
    sb = torch.rand((N + 127) // 128, K // 128, generator=gen, device="cuda") * 0.02
    common = dict(M=M, N=N, K=K, tile_m=64, tile_n=128, tile_k=128, out_dtype=out)
    outs = []
    for kw in (dict(path="tiled", block_n=256), dict()):
        fn = compile_blockscale_preshuffle_gemm(**common, **kw)
        if not kw:
            fn._cfg.max_ctas = max_ctas
            assert _plan(M, N, K, sms=0, max_ctas=max_ctas)["kernel"] == PAIR
        c = torch.full((M + 1, N), 3.0, dtype=dtype, device="cuda")
        fn(c, a, b, sa, sb, M, N, None)
        assert _lib.query_device_error() == 0
        outs.append(c)
    assert torch.equal(outs[0], outs[1])
    assert bool((outs[1][M] == 3.0).all())   # nothing beyond the last row
