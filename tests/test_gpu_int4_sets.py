"""int4 decode GEMM with one and with two sets of consumer warps: rings that wrap and that do not, an odd
number of groups, clusters whose last CTA has fewer, against the oracle."""
import pytest
import torch

from oracle import int4_ref as R
from tests.helpers import assert_close_to_oracle
from tests.test_plans import _int4_plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,split_k,sets", [(1, 128, 1152, 1, 1), (5, 128, 2176, 1, 2), (16, 256, 4352, 1, 2),
                                                (16, 384, 2176, 2, 1), (9, 256, 6272, 2, 2), (16, 128, 2816, 4, 2),
                                                (17, 128, 896, 1, 1), (20, 256, 2176, 1, 2), (32, 128, 5888, 2, 2),
                                                (32, 384, 2816, 4, 2), (31, 128, 2944, 8, 1), (33, 128, 2176, 1, 1)])
def test_int4_sets_of_warps(M, N, K, split_k, sets):
    from flydsl_b200 import _lib
    from flydsl_b200.kernels import compile_int4_weight_only_gemm, pack_int4_weight

    assert _int4_plan(M, N, K, split_k, 0)[1] == sets
    c = R.make_int4_case(M, N, K, seed=M + N + K)
    wq, st = pack_int4_weight(c["q"].cuda(), c["scales"].cuda())
    fn = compile_int4_weight_only_gemm(N=N, K=K, split_k=split_k, path="stream")
    out = torch.empty((2, M, N), dtype=torch.bfloat16, device="cuda")
    for o in out:
        fn(o, c["a"].cuda(), wq, st, M, None)
    assert _lib.query_device_error() == 0
    assert_close_to_oracle(out[0], R.int4_gemm_ref(c["a"], c["q"], c["scales"]), f"int4 {M} {N} {K} {split_k}")
    assert torch.equal(out[0], out[1])
