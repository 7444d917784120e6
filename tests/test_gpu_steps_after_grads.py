"""Steps that find something in the gradient buffer."""
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


def _same(a, b):
    for name in ("master", "exp_avg", "exp_avg_sq", "model"):
        assert torch.equal(getattr(a, name), getattr(b, name)), name


@pytest.mark.parametrize("clear", [False, True])
def test_steps_that_add_replay_a_graph(clear):
    """A loop that looks at the gradients, or clears them, before every step replays a graph for each kind of step;
    results are those of an eager engine bit for bit."""
    x, eng = _input(), [_engine(use_graph=graph) for graph in (True, False)]
    eager, real = [], eng[0]._iteration
    eng[0]._iteration = lambda *a, **kw: (eager.append(kw), real(*a, **kw))
    for i in range(4):
        for e in eng:
            e.set_input(x)
            if clear:
                e.grad.zero_()
            else:
                e.compute_grads()
        # a pass of the gradients, and the first step only: run and captured
        del eager[:]
        for e in eng:
            e.step()
        assert len(eager) == (2 if i == 0 else 0), (i, eager)
    for e in eng:
        e.step()                    # an ordinary one
        assert e.step_count == 5 and abs(e.adam_state[0].item() - 5.0) < 1e-6
        e.check_status()
    assert eng[0]._graph is not None and eng[0]._add_graph is not None
    _same(*eng)


def test_a_graph_of_adding_steps_that_fails_leaves_the_other(monkeypatch):
    import warnings
    x, eng = _input(), [_engine(use_graph=graph) for graph in (True, False)]
    real = eng[0]._iteration

    def iteration(*args, **kw):
        real(*args, **kw)
        if torch.cuda.is_current_stream_capturing() and kw["fused"] is False:
            raise torch.OutOfMemoryError("out of memory")

    monkeypatch.setattr(eng[0], "_iteration", iteration)
    with warnings.catch_warnings(record=True) as caught:
        warnings.simplefilter("always")
        for i in range(6):
            for e in eng:
                e.set_input(x)
                if i % 2:
                    e.compute_grads()
                e.step()
    assert len(caught) == 1 and eng[0]._graph is not None and eng[0]._add_graph is None and eng[0].use_graph
    _same(*eng)
