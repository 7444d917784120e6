"""What the functional calls pass on besides their tensors: the stream and the status word."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_calls_go_to_the_current_stream():
    from terapipe_b200.ops import functional as F
    assert F._stream() == torch.cuda.current_stream().cuda_stream
    side = torch.cuda.Stream()
    a, w = torch.randn(256, 4096, device="cuda").half(), torch.randn(512, 4096, device="cuda").half()
    late, out = torch.zeros_like(a), torch.empty(256, 512, device="cuda").half()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        assert F._stream() == side.cuda_stream != torch.cuda.default_stream().cuda_stream
        torch.cuda._sleep(20_000_000)
        late.copy_(a)
        F.gemm(late, w, out)
    side.synchronize()
    want = torch.empty_like(out)
    F.gemm(a, w, want)
    assert torch.equal(out, want) and F._status_ptr(a) == F.status_word(a.device).data_ptr() == F.status_word().data_ptr()
    with pytest.raises(F.KernelError):
        F.gemm(a.float(), w, out)
