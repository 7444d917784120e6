"""Column sums add up in an order that depends on sizes alone: rows of a chunk, then the chunks."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _in_order(m, chunks):
    """The kernel's fp32 sums for wide launches: of a chunk's rows eight at a time, those eight, the chunks'."""
    layers, rows, _ = m.shape
    per = (rows + chunks - 1) // chunks
    total = None
    for c in range(chunks):
        part = m[:, c * per:min(rows, (c + 1) * per)].float()
        acc = torch.zeros(layers, 8, m.shape[2], device=m.device)
        for r in range(0, part.shape[1], 8):
            n = min(8, part.shape[1] - r)
            acc[:, :n] += part[:, r:r + n]
        s = acc[:, 0].clone()
        for k in range(1, 8):
            s += acc[:, k]
        total = s if total is None else total + s
    return total


# blocks of 256 columns, on 148 SMs: 296 are two CTAs each, more take four chunks, in two CTAs up to 370 blocks
@pytest.mark.parametrize("layers,rows,widths,chunks", [
    (1, 260, (75776,), 2), (1, 260, (76032,), 4), (5, 1030, (2048, 8192, 2048, 6144), 4), (10, 701, (9472,), 4),
    (1, 515, (94976,), 4)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_order(layers, rows, widths, chunks, dtype):
    from terapipe_b200.ops import functional as F
    from terapipe_b200.ops.lib import check, cuda_lib
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the number of chunks depends on the SMs")
    gen = torch.Generator(device="cuda").manual_seed(rows)
    n, total = len(widths), sum(widths)
    mats = [torch.randn(layers, rows, w, device="cuda", generator=gen).to(dtype) for w in widths]
    out = torch.empty(layers, total, device="cuda")
    at = [sum(widths[:i]) for i in range(n)]
    P, LL, I = ctypes.c_void_p, ctypes.c_longlong, ctypes.c_int
    check(cuda_lib().tp_stage_sums(
        0 if dtype == torch.float16 else 1, n, (P * n)(*[m.data_ptr() for m in mats]), (LL * n)(*widths), (I * n)(*widths),
        (P * n)(*[out.data_ptr() + 4 * o for o in at]), rows, 0, None, 0, 0, None, None, layers,
        (LL * n)(*[rows * w for w in widths]), 0, total, 1, torch.cuda.current_stream().cuda_stream), "tp_stage_sums")
    F.check_device_status()
    assert torch.equal(out, torch.cat([_in_order(m, chunks) for m in mats], 1))
