"""What the calls for weight gradients refuse, before anything is launched."""
import pytest
import torch

from terapipe_b200.ops import functional as F
from terapipe_b200.ops.lib import KernelError, cuda_lib

K, M, N = 64, 32, 16
HALF, BF16, FP32 = torch.float16, torch.bfloat16, torch.float32


def _mats(*dtypes):
    return [torch.zeros(2, M, N, dtype=d) for d in dtypes]


@pytest.mark.parametrize("x,out", [(HALF, HALF), (HALF, BF16), (BF16, FP32), (FP32, FP32), (HALF, torch.float64)])
def test_gradient_types(x, out):
    """fp32 is stored whatever `out` is, so a 16-bit one would be overrun."""
    dy, x, out = torch.zeros(2, K, M, dtype=HALF), torch.zeros(2, K, N, dtype=x), _mats(out)[0]
    with pytest.raises(KernelError, match="float32|one type"):
        F.weight_grad(dy, x, out)


@pytest.mark.parametrize("dtypes", [(HALF, FP32, FP32, HALF), (FP32, HALF, FP32, HALF), (FP32, FP32, HALF, HALF),
                                    (FP32, FP32, FP32, FP32), (FP32, FP32, FP32, BF16)])
def test_update_types(dtypes):
    dy, x, state = torch.zeros(2, K, M, dtype=HALF), torch.zeros(2, K, N, dtype=HALF), torch.zeros(3)
    with pytest.raises(KernelError, match="float32"):
        F.weight_grad_adam(dy, x, *_mats(*dtypes), state, lr=1.0)


@pytest.mark.parametrize("layers,ldo,layer_stride", [(2, N, 0), (2, N, N), (3, N, M * N - 8), (2, 2 * N, 8), (3, 2 * N, N)])
def test_layers_that_share_elements(layers, ldo, layer_stride):
    """-1: a refused argument (anything that gets further fails otherwise, for want of a driver or of these addresses)."""
    lib, at = cuda_lib(), [4096 * i for i in range(1, 8)]
    operands = (0, at[0], M, K * M, at[1], N, K * N)
    sizes = (ldo, layer_stride, layers, M, N, K)
    assert lib.tp_wgrad(*operands, at[2], *sizes, 0, 0, None, None) == -1
    assert lib.tp_wgrad_adam(*operands, *at[2:6], *sizes, at[6], 0.1, 0.9, 0.999, 1e-8, 0.0, 1.0, 0, None, None) == -1


@pytest.mark.parametrize("ranges,layers,stride", [([(-8, 16)], 1, 0), ([(0, 8), (96, 8)], 1, 0), ([(0, 8), (32, 8)], 3, 32),
                                                  ([(0, 16)], 2, 8), ([(0, 16)], 5, 24)])
def test_ranges_outside_the_buffers(ranges, layers, stride):
    flat = [torch.zeros(100) for _ in range(4)] + [torch.zeros(100, dtype=HALF)]
    with pytest.raises(KernelError, match="do not fit"):
        F.fused_adam_ranges(*flat, torch.zeros(3), ranges, layers, stride, lr=1.0)


def test_moments_of_the_ranges_are_fp32():
    flat = [torch.zeros(100), torch.zeros(100), torch.zeros(100, dtype=HALF), torch.zeros(100), torch.zeros(100, dtype=HALF)]
    with pytest.raises(KernelError, match="float32"):
        F.fused_adam_ranges(*flat, torch.zeros(3), [(0, 8)], 1, 0, lr=1.0)
