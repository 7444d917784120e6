"""Weight gradients at each tile width, several tiles a CTA pair: the ring wraps and the accumulators change hands."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# (layers, M, N, K): the width the model takes on 148 SMs without and with Adam; K on both sides of the line for prefetches;
# rows and columns that end inside a tile.  Every shape has more than two tiles a pair at its widest.
@pytest.mark.parametrize("layers,M,N,K", [
    (9, 4136, 8, 528), (5, 8, 3952, 24), (7, 8, 2720, 3200),        # 128 with Adam (and the first without)
    (9, 8, 4152, 1032), (9, 8, 4152, 104), (9, 8, 4144, 3144),      # 192, both
    (8, 264, 2552, 128), (7, 264, 3368, 3120),                      # 256 without Adam
    (9, 1824, 4064, 24), (6, 264, 3992, 4208)])                     # 256 with Adam
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_forms(layers, M, N, K, dtype):
    from terapipe_b200.ops import functional as F
    gen = torch.Generator(device="cuda").manual_seed(M + N + K)

    def rand(*shape):
        return torch.randn(*shape, device="cuda", generator=gen)

    dy, x = rand(layers, K, M).to(dtype), rand(layers, K, N).to(dtype)
    grad = torch.full((layers, M, N), float("nan"), device="cuda")
    F.weight_grad(dy, x, grad)
    for l in range(layers):
        exact = dy[l].double().t() @ x[l].double()
        # fp32 sums of K products of magnitude about 1, whose results are about sqrt(K)
        assert ((grad[l] - exact).norm() / exact.norm()).item() < 1e-6 * K ** 0.5
    base = rand(layers, M, N)
    added = base.clone()
    F.weight_grad(dy, x, added, accumulate=True)
    assert torch.equal(added, base + grad)      # one fp32 addition an element
    master, m, v = rand(layers, M, N), rand(layers, M, N), rand(layers, M, N).abs_()
    model = master.to(dtype)
    want = [t.clone().view(-1) for t in (master, m, v, model)]
    state = torch.tensor([3.0, 1 - 0.9 ** 3, 1 - 0.999 ** 3], device="cuda")
    kw = dict(lr=1e-2, weight_decay=0.01, grad_scale=0.125)
    F.weight_grad_adam(dy, x, master, m, v, model, state, **kw)
    F.fused_adam(grad.view(-1), *want, state, **kw)
    F.check_device_status()
    for got, w in zip((master, m, v, model), want):
        assert torch.equal(got.view(-1), w)
