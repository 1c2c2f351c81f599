"""1x128 quantiser over rows in routing order: rows with a route as the plain quantiser gives them, the others (and
their scales) untouched."""
import pytest
import torch

from flydsl_b200 import _lib
from flydsl_b200.utils import moe_sorting, quant_1x128, route_topk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,E,k,block,cols,dtype", [(1, 8, 1, 8, 128, torch.float16), (37, 16, 4, 32, 1152, torch.bfloat16),
                                                    (300, 32, 6, 128, 2048, torch.float16),
                                                    (5, 256, 8, 16, 256, torch.bfloat16)])
def test_rows_with_a_route_only(T, E, k, block, cols, dtype):
    g = torch.Generator(device="cuda").manual_seed(T + cols)
    ids, w = route_topk(torch.randn(T, E, generator=g, device="cuda"), k)
    sid, _, _, npp = moe_sorting(ids, w, num_experts=E, block_size=block)
    L = sid.numel()
    x = torch.randn(L, cols, generator=g, device="cuda").to(dtype)
    q = torch.full((L, cols), 0x5A, dtype=torch.uint8, device="cuda")
    s = torch.full((cols // 128, L), -7.0, device="cuda")
    code = _lib.F16 if dtype == torch.float16 else _lib.BF16
    _lib.check(_lib.load().flyb200_quant_1x128_routes(x.data_ptr(), q.data_ptr(), s.data_ptr(), npp.data_ptr(),
                                                      sid.data_ptr(), T, k, L, cols, code, _lib.stream_handle(None)))
    want_q, want_s = quant_1x128(x)
    used = ((sid & 0xFFFFFF) < T) & (torch.arange(L, device="cuda") < npp[0])
    assert int(used.sum()) == T * k
    assert torch.equal(q[used], want_q.view(torch.uint8)[used]) and torch.equal(s[:, used], want_s[:, used])
    assert bool((q[~used] == 0x5A).all()) and bool((s[:, ~used] == -7.0).all())


def test_bad_arguments():
    one = torch.zeros(128, dtype=torch.float16, device="cuda")
    p, st = one.data_ptr(), _lib.stream_handle(None)
    for sid, T, k in ((None, 1, 1), (p, 0, 1), (p, 1, 0), (p, 1, 256)):
        with pytest.raises(ValueError):
            _lib.check(_lib.load().flyb200_quant_1x128_routes(p, p, p, p, sid, T, k, 1, 128, _lib.F16, st))
