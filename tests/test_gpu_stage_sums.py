"""Column sums of one and of several layers, both types, at each width of block and number of chunks."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


# narrow blocks (1 and 8 chunks), wide ones: 8, 4, 2 chunks as they fill the SMs, 2 for up to five CTAs an SM, 4 past that
@pytest.mark.parametrize("layers,rows,widths", [(1, 9, (72,)), (3, 130, (264, 8)), (2, 2500, (776, 1032)),
                                                (1, 2100, (12288,)), (3, 1100, (12288, 2056)), (5, 1030, (16384, 2048)),
                                                (1, 1030, (92160,)), (6, 1030, (16384,)), (5, 1030, (24576,))])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_sums(layers, rows, widths, dtype):
    from terapipe_b200.ops import functional as F
    from terapipe_b200.ops.lib import check, cuda_lib
    gen = torch.Generator(device="cuda").manual_seed(rows + layers)
    n, total = len(widths), sum(widths)
    mats = [torch.randn(layers, rows, w, device="cuda", generator=gen).to(dtype) for w in widths]
    out = torch.randn(layers, total, device="cuda", generator=gen)
    want = out.double() + torch.cat([m.double().sum(1) for m in mats], 1)
    at = [sum(widths[:i]) for i in range(n)]
    P, LL, I = ctypes.c_void_p, ctypes.c_longlong, ctypes.c_int
    check(cuda_lib().tp_stage_sums(
        0 if dtype == torch.float16 else 1, n, (P * n)(*[m.data_ptr() for m in mats]), (LL * n)(*widths), (I * n)(*widths),
        (P * n)(*[out.data_ptr() + 4 * o for o in at]), rows, 0, None, 0, 0, None, None, layers,
        (LL * n)(*[rows * w for w in widths]), 0, total, 0, torch.cuda.current_stream().cuda_stream), "tp_stage_sums")
    F.check_device_status()
    # fp32 sums of `rows` values of magnitude 1
    assert ((out.double() - want).norm() / want.norm()).item() < 2e-6 * max(1.0, rows ** 0.5 / 8)
