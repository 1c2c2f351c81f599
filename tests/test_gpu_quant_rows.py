"""The quantisers where a row is dealt out to several warps (few rows), held by 32 to 256 threads (whole
rows), or too long for that: bit for bit the torch quantiser, special values included."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rows(rows, cols, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    x = (torch.randn(rows, cols, generator=g) * 3).to(dtype)
    x[0, : cols // 2] = 0.0                      # a zero group / half a zero row
    x[0, 1] = -0.0
    x[-1, 3], x[-1, cols - 1] = float("nan"), float("-inf")
    x[rows // 2, cols // 2] = float("inf")
    x[rows // 2, 0] = -float("nan")
    return x


@pytest.mark.parametrize("rows,cols", [(1, 128), (3, 1024), (1, 1152), (32, 7168), (777, 2304), (20000, 256)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_quant_1x128(rows, cols, dtype):
    from flydsl_b200.utils import pertoken_quant, quant_1x128

    x = _rows(rows, cols, dtype, rows + cols)
    q, s = quant_1x128(x.cuda())
    want_q, want_s = pertoken_quant(x.float().view(-1, 128))
    assert torch.equal(q.cpu().view(torch.uint8), want_q.view(rows, cols).view(torch.uint8))
    assert torch.equal(s.cpu().t().contiguous().view(-1), want_s.view(-1))


# 8 values; one chunk short of and one beyond what 32, 64, 128 and 256 threads hold; two passes
@pytest.mark.parametrize("cols", [8, 2048, 2056, 4096, 4104, 8200, 16384, 16392])
@pytest.mark.parametrize("rows", [1, 5, 700, 6000])
def test_quant_pertoken(rows, cols):
    from flydsl_b200.utils import pertoken_quant, quant_pertoken

    if rows == 6000 and cols > 4104:
        pytest.skip("the same kernel as with 700 rows")
    for dtype in (torch.bfloat16, torch.float16):
        x = _rows(rows, cols, dtype, rows + cols)
        q, s = quant_pertoken(x.cuda())
        want_q, want_s = pertoken_quant(x)
        assert torch.equal(q.cpu().view(torch.uint8), want_q.view(torch.uint8))
        assert torch.equal(s.cpu(), want_s.view(-1))
        # a row count known on the device only: the other rows stay as they are
        n = torch.tensor([rows - 1], dtype=torch.int32, device="cuda")
        out = torch.zeros((rows, cols), dtype=torch.uint8, device="cuda").view(torch.float8_e4m3fn)
        q, _ = quant_pertoken(x.cuda(), n, out=out)
        assert torch.equal(q.cpu().view(torch.uint8)[: rows - 1], want_q.view(torch.uint8)[: rows - 1])
        assert not q.view(torch.uint8)[rows - 1].any()
