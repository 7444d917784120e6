"""Whatever writes to the gradient buffer between steps counts, for weights as for biases."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _engine(**kw):
    from terapipe_b200.models import TransformerConfig
    from terapipe_b200.runtime.engine import StageEngine
    cfg = TransformerConfig(batch_size=2, seq_len=64, n_layers=2, embedding_dim=256,
                            num_attention_heads=4, n_devices=1)
    return StageEngine(cfg, [2], [64], lr=1e-3, **kw)


def _input():
    return torch.randn(64, 2, 256, generator=torch.Generator().manual_seed(3))


def _write(e, how, held):
    """Something added to a weight's gradient and to a bias's, in ways torch's version counter does not see."""
    from terapipe_b200.ops import functional as F
    gen = torch.Generator(device="cuda").manual_seed(9)
    dy, x = (torch.randn(64, n, device="cuda", generator=gen).half() for n in (1024, 256))
    w, b = "fc1.weight", "fc1.bias"
    if how == "data":
        e.param(1, w, e.grad.data).add_(0.5)
        e.param(1, b, e.grad.data).add_(0.25)
    elif how == "kernels":
        F.weight_grad(dy, x, e.param(1, w, e.grad), accumulate=True)
        F.gemm(dy, x, e.param(0, w, e.grad), a_mn=True, b_mn=True, accumulate=True)
        F.colsum(dy, e.param(1, b, e.grad))
    else:                                        # a view taken once
        held[0].add_(0.5)
        held[1].data.add_(0.25)


@pytest.mark.parametrize("how", ["data", "kernels", "held"])
@pytest.mark.parametrize("use_graph", [False, True])
def test_writes_count(how, use_graph):
    x, eng = _input(), [_engine(use_graph=use_graph) for _ in range(2)]
    eng[1]._adam_in_products = False             # always adds to what the buffer holds
    held = [[e.param(1, n, e.grad) for n in ("fc1.weight", "fc1.bias")] if how == "held" else None for e in eng]
    for i in range(6):
        for e, h in zip(eng, held):
            e.set_input(x)
            if i % 2:
                _write(e, how, h)
            e.step()
    for name in ("master", "exp_avg", "exp_avg_sq", "model"):
        assert torch.equal(getattr(eng[0], name), getattr(eng[1], name)), name
    assert eng[0]._updates_in_products == (how != "held")
    for e in eng:
        e.check_status()
        assert e.grad.abs().max().item() == 0


@pytest.mark.parametrize("use_graph", [False, True])
def test_engine_made_in_inference_mode(use_graph):
    x, want = _input(), _engine(use_graph=use_graph)
    with torch.inference_mode():
        got = _engine(use_graph=use_graph)
        for i in range(5):
            for e in (want, got):
                e.set_input(x)
                if i == 3:
                    e.compute_grads()
                e.step()
        for name in ("master", "exp_avg", "exp_avg_sq", "model"):
            assert torch.equal(getattr(want, name), getattr(got, name)), name
        got.check_status()


@pytest.mark.parametrize("kind", [dict(launch_plan=True, segment_graphs=False), dict(launch_plan=False, segment_graphs=True)])
def test_writes_count_in_replayed_segments(kind):
    """Plans and segment graphs keep the adding products apart from those that update."""
    x, eng = _input(), [_engine(use_graph=False, merge_slices=False, **k) for k in (kind, dict(segment_graphs=False))]
    assert (eng[0]._plan is not None) == kind["launch_plan"] and (eng[0]._seg_graphs is not None) == kind["segment_graphs"]
    for i in range(12):
        for e in eng:
            e.set_input(x)
            if i % 3 == 1:
                _write(e, "kernels", None)
            if i % 3 == 2:
                e.compute_grads()
            e.step()
    for name in ("master", "exp_avg", "exp_avg_sq", "model"):
        assert torch.equal(getattr(eng[0], name), getattr(eng[1], name)), name
    for e in eng:
        e.check_status()
        assert e.grad.abs().max().item() == 0
