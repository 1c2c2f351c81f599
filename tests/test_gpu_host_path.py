"""What a call looks up on the host: the current stream's handle and the device of its tensors."""
import pytest
import torch

from flydsl_b200 import _lib


@pytest.mark.gpu
def test_stream_handle_and_device_guard_follow_torch():
    side = torch.cuda.Stream()
    assert _lib.stream_handle(None) == torch.cuda.current_stream().cuda_stream
    with torch.cuda.stream(side):
        assert _lib.stream_handle(None) == side.cuda_stream == _lib.stream_handle(side)
    assert _lib.stream_handle(None) == torch.cuda.current_stream().cuda_stream
    for index in range(torch.cuda.device_count()):
        with _lib.device_guard(torch.empty(1, device=f"cuda:{index}")):
            assert torch.cuda.current_device() == index
            assert _lib.stream_handle(None) == torch.cuda.current_stream().cuda_stream
        assert torch.cuda.current_device() == 0


@pytest.mark.skipif(torch.cuda.is_available(), reason="needs a machine without a GPU")
def test_current_stream_without_a_gpu_is_torchs_error():
    with pytest.raises((RuntimeError, AssertionError)):
        _lib.stream_handle(None)
