"""The optimizer's numbers of a step are those set when the step is taken."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_launch_plan_follows_lr_and_loss_scale():
    """A step replayed from a recorded plan uses the learning rate and loss scale of now, for weights as for biases."""
    from terapipe_b200.models import TransformerConfig
    from terapipe_b200.runtime.engine import StageEngine
    cfg = TransformerConfig(batch_size=2, seq_len=64, n_layers=2, embedding_dim=256,
                            num_attention_heads=4, n_devices=1)
    gen = torch.Generator().manual_seed(5)
    xs = [torch.randn(64, 2, 256, generator=gen) for _ in range(6)]
    engines = []
    for plan in (False, True):
        eng = StageEngine(cfg, [2], [24, 40], use_graph=False, lr=1e-3, launch_plan=plan, segment_graphs=False,
                          merge_slices=False)
        assert (eng._plan is not None) == plan
        for i, x in enumerate(xs):
            if i == 2:
                eng.lr = 3e-3
            if i == 4:
                eng.lr, eng.loss_scale = 5e-4, 2 * eng.loss_scale
            eng.set_input(x)
            eng.step()
        eng.check_status()
        engines.append(eng)
    assert engines[1]._plan.replayed > 0
    for name in ("master", "exp_avg", "exp_avg_sq", "model"):
        assert torch.equal(getattr(engines[0], name), getattr(engines[1], name)), name
