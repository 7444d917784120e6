"""Adam in the epilogue of the weight-gradient products."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# tiles of 128, 192 and 256 columns; rows and columns that end inside a tile and inside a 32 x 32 chunk, K of
# less than a step and of many, fewer tiles than CTA pairs and several waves
@pytest.mark.parametrize("layers,M,N,K", [(1, 8, 8, 8), (3, 256, 256, 256), (2, 1000, 776, 300), (5, 136, 2056, 72),
                                          (1, 2304, 768, 4096), (4, 2048, 1032, 1024), (2, 2048, 5120, 640),
                                          (1, 5120, 2560, 8192)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_update_equals_gradient_then_adam(layers, M, N, K, dtype):
    """The same fp32 sums and the same update as the product stored and a pass over it: equal bit for bit.  The
    matrices are cut out of wider ones, whose other columns stay as they are."""
    from terapipe_b200.ops import functional as F
    gen = torch.Generator(device="cuda").manual_seed(M + N + K)

    def rand(*shape):
        return torch.randn(*shape, device="cuda", generator=gen)

    a, b = rand(layers, K, M + 8).to(dtype)[:, :, :M], rand(layers, K, N).to(dtype)
    full = [rand(layers, M, N + 16) for _ in range(3)]
    full[2].abs_()
    full.append(full[0].to(dtype))
    want = [t.clone() for t in full]
    state = torch.tensor([3.0, 1 - 0.9 ** 3, 1 - 0.999 ** 3], device="cuda")
    kw = dict(lr=1e-2, weight_decay=0.01, grad_scale=0.125)
    F.weight_grad_adam(a, b, *(t[:, :, 8:N + 8] for t in full), state, **kw)
    grad = torch.full((layers, M, N), float("nan"), device="cuda")
    F.weight_grad(a, b, grad)
    exact = torch.einsum("lkm,lkn->lmn", a.double(), b.double())
    # fp32 sums of K products of magnitude about 1, whose results are about sqrt(K)
    assert ((grad - exact).norm() / exact.norm()).item() < 1e-6 * K ** 0.5
    twice = grad.clone()
    F.weight_grad(a, b, twice, accumulate=True)
    assert torch.equal(twice, 2 * grad)
    flat = [t[:, :, 8:N + 8].contiguous().view(-1) for t in want]
    F.fused_adam(grad.view(-1), *flat, state, **kw)
    F.check_device_status()
    for got, t, f in zip(full, want, flat):
        t[:, :, 8:N + 8] = f.view(layers, M, N)
        assert torch.equal(got, t)


@pytest.mark.parametrize("layers,rows,widths", [(1, 7, (8,)), (3, 33, (256, 264)), (24, 256, (256, 1024, 256, 768)),
                                                (2, 5000, (2048, 8, 776))])
def test_sums_of_all_layers_in_one_launch(layers, rows, widths):
    """Column sums and LayerNorm folds of several layers, added and assigned.  fp32 sums of `rows` values of
    magnitude 1: 1e-6 sqrt(rows) of the result's magnitude sqrt(rows)."""
    import ctypes
    from terapipe_b200.ops import functional as F
    from terapipe_b200.ops.lib import check, cuda_lib
    torch.manual_seed(rows)
    H, parts, n = 264, 5, len(widths)
    total = sum(widths) + 2 * H + 8
    mats = [torch.randn(layers, rows, w, device="cuda").half() for w in widths]
    at = [sum(widths[:i]) for i in range(n + 1)]
    P, LL, I = ctypes.c_void_p, ctypes.c_longlong, ctypes.c_int
    for assign in (0, 1):
        slots = torch.randn(layers, parts, 2, H, device="cuda")
        out = torch.ones(layers, total, device="cuda")
        want = torch.ones_like(out) - assign
        want[:, total - 8:] = 1
        for m, o, w in zip(mats, at, widths):
            want[:, o:o + w] += m.double().sum(1).float()
        want[:, at[n]:at[n] + 2 * H] += slots.sum(1).reshape(layers, 2 * H)
        base = out.data_ptr()
        check(cuda_lib().tp_stage_sums(
            0, n, (P * n)(*[m.data_ptr() for m in mats]), (LL * n)(*widths), (I * n)(*widths),
            (P * n)(*[base + 4 * o for o in at[:n]]), rows, 1, (P * 1)(slots.data_ptr()), parts, H,
            (P * 1)(base + 4 * at[n]), (P * 1)(base + 4 * (at[n] + H)), layers, (LL * n)(*[rows * w for w in widths]),
            parts * 2 * H, total, assign, torch.cuda.current_stream().cuda_stream), "tp_stage_sums")
        assert ((out - want).abs().max() / (1 + rows ** 0.5)).item() < 1e-6 * (10 + rows ** 0.5)
        assert slots.abs().max().item() == 0.0
    F.check_device_status()


@pytest.mark.parametrize("use_graph", [False, True])
def test_gradients_left_in_the_buffer_count(use_graph):
    """A step after compute_grads() adds to what that left, and the step after it is an ordinary one."""
    from terapipe_b200.models import TransformerConfig
    from terapipe_b200.runtime.engine import StageEngine
    cfg = TransformerConfig(batch_size=2, seq_len=64, n_layers=2, embedding_dim=256,
                            num_attention_heads=4, n_devices=1)
    x = torch.randn(64, 2, 256, generator=torch.Generator().manual_seed(3))
    eng = [StageEngine(cfg, [2], [64], lr=1e-3, use_graph=use_graph) for _ in range(2)]
    eng[1]._adam_in_products = False
    for _ in range(3):
        for e in eng:
            e.set_input(x)
            e.step()
    for e in eng:
        e.compute_grads()
        assert e.grad.abs().max().item() > 0
        e.step()                    # the sum of two gradients
        assert e.grad.abs().max().item() == 0
        e.step()
        e.check_status()
        assert e.step_count == 5 and abs(e.adam_state[0].item() - 5.0) < 1e-6
        assert e.grad.abs().max().item() == 0
    for name in ("master", "exp_avg", "exp_avg_sq", "model"):
        assert torch.equal(getattr(eng[0], name), getattr(eng[1], name)), name
    assert (eng[0]._graph is not None) == use_graph
