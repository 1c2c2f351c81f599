"""int4 decode GEMM on tcgen05 (weights dequantised into tensor memory): rings that wrap and that do not, odd and
single groups, clusters whose last CTA has fewer, every token-column width and its edges, all nibbles."""
import pytest
import torch

from oracle import int4_ref as R
from tests.helpers import assert_close_to_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,split_k", [
    (1, 128, 128, 1), (16, 128, 256, 1), (16, 256, 384, 1),      # one, two and three groups
    (5, 128, 1152, 1), (16, 384, 4224, 1), (15, 128, 10240, 1),  # the ring wraps, odd numbers of groups, few slots
    (17, 128, 1152, 1), (32, 256, 3968, 2), (31, 128, 2176, 8),
    (33, 128, 128, 1), (64, 256, 2944, 3), (63, 128, 4992, 1), (48, 384, 2176, 4),
    (16, 128, 2304, 7), (2, 4736, 1024, 8),                      # last CTA with fewer groups; more than one wave
    (16, 128, 49152, 1),                                         # scales leave room for a whole-SM ring only
])
def test_int4_tensor_vs_oracle(M, N, K, split_k):
    from flydsl_b200 import _lib
    from flydsl_b200.kernels import compile_int4_weight_only_gemm, pack_int4_weight

    c = R.make_int4_case(M, N, K, seed=M + N + K)
    c["q"][0, :16] = torch.arange(-8, 8, dtype=torch.int8)       # every nibble in every position of a word
    for i in range(1, 8):
        c["q"][i, :16] = torch.roll(c["q"][0, :16], i)
    wq, st = pack_int4_weight(c["q"].cuda(), c["scales"].cuda())
    fn = compile_int4_weight_only_gemm(N=N, K=K, split_k=split_k, path="tensor")
    out = torch.full((2, M + 1, N), 5.0, dtype=torch.bfloat16, device="cuda")
    for o in out:
        fn(o[:M], c["a"].cuda(), wq, st, M, None)
    assert _lib.query_device_error() == 0
    assert_close_to_oracle(out[0][:M], R.int4_gemm_ref(c["a"], c["q"], c["scales"]), f"int4 {M} {N} {K} {split_k}")
    assert torch.equal(out[0], out[1]) and bool((out[:, M] == 5.0).all())


def test_int4_tensor_weights_are_exact():
    """One-hot activations pick single weights: q * scale, exactly (bf16 scale times a small integer, rounded once)."""
    from flydsl_b200.kernels import compile_int4_weight_only_gemm, pack_int4_weight

    N, K = 256, 256
    g = torch.Generator().manual_seed(0)
    q = torch.randint(-8, 8, (N, K), generator=g, dtype=torch.int8)
    scales = (torch.rand(N, K // 128, generator=g) + 0.5).to(torch.bfloat16)
    wq, st = pack_int4_weight(q.cuda(), scales.cuda())
    fn = compile_int4_weight_only_gemm(N=N, K=K, path="tensor")
    want = (q.view(N, K // 128, 128).float() * scales.float().unsqueeze(-1)).to(torch.bfloat16).view(N, K).t()
    for k0 in range(0, K, 64):
        a = torch.zeros(64, K, dtype=torch.bfloat16)
        a[torch.arange(64), k0 + torch.arange(64)] = 1.0
        out = torch.empty(64, N, dtype=torch.bfloat16, device="cuda")
        fn(out, a.cuda(), wq, st, 64, None)
        assert torch.equal(out.cpu(), want[k0:k0 + 64])
