"""What the int4 GEMM refuses before anything is launched. Host code: no GPU is needed."""
import ctypes

import pytest


def test_operands_of_bulk_copies_are_16_byte_aligned():
    """Tokens, packed weights and group scales are all fetched by copies that start on a 16-byte boundary. The
    addresses are never dereferenced: every call here is refused."""
    from flydsl_b200 import _lib

    lib, aligned = _lib.load(), 1 << 20
    for path in (0, 1, 2):
        cfg = _lib.GemmCfg(0, 0, path, 0)
        for operand in ("a", "wq", "scales_t"):
            for offset in (2, 4, 8, 14):
                p = {name: aligned + (offset if name == operand else 0) for name in ("a", "wq", "scales_t")}
                with pytest.raises(ValueError, match="16-byte aligned"):
                    _lib.check(lib.flyb200_int4_gemm(aligned, p["a"], p["wq"], p["scales_t"], 16, 256, 512,
                                                     ctypes.byref(cfg), None))


@pytest.mark.parametrize("change,message", [
    (dict(wq=lambda t: t[:-1]), "wq must"), (dict(wq=lambda t: t.transpose(0, 1)), "wq must"),
    (dict(scales=lambda t: t.float()), "scales_t must"), (dict(scales=lambda t: t[:, :-128]), "scales_t must"),
    (dict(scales=lambda t: t.t()), "scales_t must"), (dict(), "CUDA tensors")])
def test_launcher_refuses_weights_that_the_kernel_would_read_beyond(change, message):
    import torch

    from flydsl_b200.kernels import compile_int4_weight_only_gemm

    M, N, K = 4, 256, 512
    wq = torch.zeros(K // 128, N // 8, 4, 8, 16, dtype=torch.uint8)
    scales = torch.ones(K // 128, N, dtype=torch.bfloat16)
    a, c = torch.zeros(M, K, dtype=torch.bfloat16), torch.zeros(M, N, dtype=torch.bfloat16)
    keep = lambda t: t  # noqa: E731
    with pytest.raises(ValueError, match=message):
        compile_int4_weight_only_gemm(N=N, K=K)(c, a, change.get("wq", keep)(wq), change.get("scales", keep)(scales), M)
