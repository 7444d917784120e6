"""Kernels that start before their predecessor has ended give what they give one after the other."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def set_pdl():
    from terapipe_b200.ops.lib import cuda_lib
    before = cuda_lib().tp_pdl_enabled()
    yield cuda_lib().tp_set_pdl
    cuda_lib().tp_set_pdl(before)


# dQ beside a dK/dV that takes far longer (first slice), far less long (last slice), and about as long; one and two
# rounds of CTAs, which wait for each other's TMEM
@pytest.mark.parametrize("b,h,D,L,t,c", [(2, 4, 64, 2048, 64, 0), (1, 12, 64, 1024, 77, 940), (2, 8, 128, 512, 512, 0),
                                         (4, 40, 128, 640, 128, 256), (3, 30, 64, 300, 150, 100)])
def test_attention_backward_in_a_row(b, h, D, L, t, c, set_pdl):
    """Every round has new gradients and is read by a product that follows at once; the buffers are the same."""
    from terapipe_b200.ops import functional as F
    gen = torch.Generator(device="cuda").manual_seed(L + t)

    def rand(*shape):
        return torch.randn(*shape, device="cuda", generator=gen).half()

    W = h * D
    qkv, do0, w_o, w_qkv = rand(L, b, 3 * W), rand(L * b, W), rand(W, W) * W ** -0.5, rand(256, 3 * W) * W ** -0.5
    grads = [rand(t * b, W) for _ in range(12)]
    o, lse = torch.empty(L * b, W, device="cuda").half(), torch.empty(b * h, L, device="cuda")
    F.attn_fwd(qkv, b, h, D, L, 0, o, lse)
    first = (o.float() * do0.float()).view(L, b, h, D).sum(-1).permute(1, 2, 0).reshape(b * h, L).contiguous()
    rows = slice(c * b, (c + t) * b)
    out = []
    for pdl in (0, 1):
        set_pdl(pdl)
        d_o, delta = do0.clone(), first.clone()
        dqkv = torch.full((t * b, 3 * W), float("nan"), device="cuda").half()
        outs = [torch.empty(t * b, 256, device="cuda").half() for _ in grads]
        torch.cuda.synchronize()
        torch.cuda._sleep(3_000_000)       # the launches below queue up behind it
        for g, x in zip(grads, outs):
            F.gemm(g, w_o, d_o[rows])
            F.attn_bwd(qkv, b, h, D, t, c, L, o[rows], d_o, lse, delta, dqkv)
            F.gemm(dqkv, w_qkv, x)
        F.check_device_status()
        out.append(torch.cat([x.view(-1) for x in outs + [dqkv]]))
    assert not out[0].isnan().any() and torch.equal(out[0], out[1])


# all four products on the chip at once, one wave each, several; gradients added and assigned, weights updated
@pytest.mark.parametrize("layers,H,heads,L", [(1, 128, 2, 40), (3, 256, 4, 512), (2, 1024, 16, 136), (5, 1600, 25, 64)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_weight_gradients_in_a_row(layers, H, heads, L, dtype, set_pdl):
    from terapipe_b200.models import TransformerConfig
    from terapipe_b200.runtime.engine import StageEngine
    cfg = TransformerConfig(batch_size=2, seq_len=L, n_layers=layers, embedding_dim=H, num_attention_heads=heads,
                            n_devices=1)
    gen = torch.Generator(device="cuda").manual_seed(H + L)
    xs = [torch.randn(L, 2, H, device="cuda", generator=gen).to(dtype) for _ in range(4)]
    out = []
    for pdl in (0, 1):
        set_pdl(pdl)
        eng = StageEngine(cfg, [2], [L], dtype=dtype, use_graph=False, lr=1e-3, loss_scale=1024.0)
        got = []
        eng.set_input(xs[0])
        eng.step()
        torch.cuda.synchronize()
        torch.cuda._sleep(3_000_000)       # the launches below queue up behind it
        for x in xs:
            eng.set_input(x)
            eng.compute_grads()            # assigned
            got.append(eng.grad.clone())
            eng.step()                     # added to those, which the next product's weights come from
            eng.step()                     # weights updated in the products
            got += [eng.master.clone(), eng.exp_avg_sq.clone(), eng.model.clone().float(), eng.grad.clone()]
        eng.check_status()
        out.append(got)
    assert all(torch.equal(a, b) for a, b in zip(*out))
    assert out[0][0].abs().max() > 0 and not any(t.isnan().any() for t in out[0])
