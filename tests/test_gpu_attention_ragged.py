"""Attention backward where slices start and the sequence ends inside a block of 64 positions."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,L,slices", [
    (64, 193, [77, 51, 65]),            # nothing a multiple of four
    (128, 259, [1, 130, 128]),          # a slice of one position, starts at 1 and 131
    (128, 66, [66]),                    # the sequence ends two positions into a block
    (64, 130, [3, 127]),
])
def test_slices_anywhere_in_the_sequence(D, L, slices):
    """Slices against one whole-sequence call and against fp32 autograd.  Only the rounding of P, dS
    and of the results to fp16 differs: a few times 2^-11."""
    from terapipe_b200.ops import functional as F
    torch.manual_seed(3)
    b, h = 2, 3
    qkv = torch.randn(L, b, h * 3 * D, device="cuda", dtype=torch.float16)
    g = torch.randn(L * b, h * D, device="cuda", dtype=torch.float16)
    o = torch.empty(L * b, h * D, device="cuda", dtype=torch.float16)
    lse = torch.full((b * h, L), float("nan"), device="cuda")
    delta = torch.full((b * h, L), float("nan"), device="cuda")
    dqkv = torch.full((L * b, h * 3 * D), float("nan"), device="cuda", dtype=torch.float16)
    c = 0
    for t in slices:
        F.attn_fwd(qkv, b, h, D, t, c, o[c * b:(c + t) * b], lse)
        c += t
    do = torch.full_like(g, float("nan"))
    for t in reversed(slices):
        c -= t
        do[c * b:(c + t) * b] = g[c * b:(c + t) * b]
        F.attn_bwd(qkv, b, h, D, t, c, L, o[c * b:(c + t) * b], do, lse, delta, dqkv[c * b:(c + t) * b])
    F.check_device_status()
    x = qkv.float().requires_grad_()
    q, k, v = (x.view(L, b, h, 3, D)[:, :, :, i].permute(1, 2, 0, 3) for i in range(3))
    ref = torch.nn.functional.scaled_dot_product_attention(q, k, v, is_causal=True)
    ref = ref.permute(2, 0, 1, 3).reshape(L * b, h * D)
    ref.backward(g.float())
    assert ((o.float() - ref).norm() / ref.norm()).item() < 2e-3
    got, want = dqkv.view(L, b, h, 3, D).float(), x.grad.view(L, b, h, 3, D)
    for w in range(3):
        assert ((got[:, :, :, w] - want[:, :, :, w]).norm() / want[:, :, :, w].norm()).item() < 4e-3, "qkv"[w]
