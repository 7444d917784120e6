"""Attention at the edges of its tiles: 128-row query tiles (256 per CTA), 64-row streamed blocks, the
key split of a last single tile, and rows whose first block of the split lies beyond the diagonal."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(qkv, b, h, D, t, c, d_o):
    """fp64 output, log2-sum-exp and d(qkv) of the slice [c, c + t) and everything after it."""
    L = qkv.shape[0]
    x = qkv.double().view(L, b, h, 3, D).requires_grad_()
    q, k, v = (x[:, :, :, i].permute(1, 2, 0, 3) for i in range(3))
    s = q @ k.transpose(-1, -2) / math.sqrt(D)
    s = s.masked_fill(torch.ones(L, L, device=qkv.device, dtype=torch.bool).triu(1), float("-inf"))
    o = (s.softmax(-1) @ v).permute(2, 0, 1, 3).reshape(L * b, h * D)
    o.backward(d_o.double())
    lse = torch.logsumexp(s.detach(), -1).reshape(b * h, L) / math.log(2.0)
    return o.detach(), lse, x.grad.reshape(L * b, 3 * h * D)


def _rel(a, ref):
    return ((a.double() - ref).norm() / ref.norm()).item()


# (L, b, h, D, t, c): tile edges +- 1, splits of one, two and many blocks, odd batch and heads
CASES = [(64, 1, 1, 64, 1, 0), (65, 1, 2, 128, 1, 64), (130, 2, 1, 64, 128, 1), (129, 1, 3, 128, 129, 0),
         (257, 1, 2, 64, 257, 0), (255, 2, 2, 128, 255, 0), (400, 1, 2, 128, 256, 100),
         (400, 3, 1, 64, 385, 15), (600, 1, 5, 128, 127, 390), (320, 1, 17, 64, 100, 31),
         (513, 1, 2, 128, 384, 129), (200, 1, 2, 64, 65, 63)]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("L,b,h,D,t,c", CASES)
def test_slice_forward_and_backward(L, b, h, D, t, c, dtype):
    from terapipe_b200.ops import functional as F
    g = torch.Generator(device="cuda").manual_seed(L + t + c)
    qkv = torch.randn(L, b, 3 * h * D, device="cuda", generator=g).to(dtype)
    # a few large scores, so that the running maximum moves between blocks
    qkv[::37] *= 3
    d_o = torch.randn(L * b, h * D, device="cuda", generator=g).to(dtype)
    ref_o, ref_lse, ref_d = _reference(qkv, b, h, D, t, c, d_o)
    rows = slice(c * b, (c + t) * b)
    o = torch.empty(t * b, h * D, device="cuda", dtype=dtype)
    lse = ref_lse.float().contiguous()
    lse[:, c:c + t] = float("nan")
    F.attn_fwd(qkv, b, h, D, t, c, o, lse)
    F.check_device_status()
    # P, dS and the results are rounded to 16 bits (2^-11, 2^-8); sums are fp32
    tol = 2e-3 if dtype == torch.float16 else 1.2e-2
    assert _rel(o, ref_o[rows]) < tol
    assert (lse[:, c:c + t].double() - ref_lse[:, c:c + t]).abs().max().item() < 1e-4
    delta = (ref_o * d_o.double()).view(L, b, h, D).sum(-1).permute(1, 2, 0).reshape(b * h, L).float().contiguous()
    dqkv = torch.empty(t * b, 3 * h * D, device="cuda", dtype=dtype)
    F.attn_bwd(qkv, b, h, D, t, c, L, o, d_o, lse, delta, dqkv)
    F.check_device_status()
    assert _rel(dqkv, ref_d[rows]) < 2 * tol


def test_delta_of_an_output_that_is_only_4_byte_aligned():
    from terapipe_b200.ops import functional as F
    torch.manual_seed(3)
    b, h, D, t = 1, 2, 64, 96
    qkv = torch.randn(t, b, 3 * h * D, device="cuda", dtype=torch.float16)
    d_o = torch.randn(t * b, h * D, device="cuda", dtype=torch.float16)
    o, lse = torch.empty(t * b, h * D, device="cuda", dtype=torch.float16), torch.empty(b * h, t, device="cuda")
    F.attn_fwd(qkv, b, h, D, t, 0, o, lse)
    shifted = torch.empty(t * b * h * D + 2, device="cuda", dtype=torch.float16)[2:].view(t * b, h * D)
    shifted.copy_(o)
    out = []
    for src in (o, shifted):
        delta, dqkv = torch.empty(b * h, t, device="cuda"), torch.empty(t * b, 3 * h * D, device="cuda", dtype=torch.float16)
        F.attn_bwd(qkv, b, h, D, t, 0, t, src, d_o, lse, delta, dqkv)
        out.append((delta, dqkv))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
