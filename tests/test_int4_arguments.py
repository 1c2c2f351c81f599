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
