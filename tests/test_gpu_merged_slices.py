"""A stage without pipeline neighbours walks all rows at once; slices give the same training."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch_slices,seq_slices", [([3], [24, 40, 64]), ([2, 1], [128]),
                                                     ([1, 2], [37, 91])])
def test_merged_pass_equals_slice_by_slice(batch_slices, seq_slices):
    """fp16 rounding of 2 layers' activations apart (rows come from the same kernels; sums over rows
    are split differently), the merged engine and one that was told to keep its slices agree."""
    from terapipe_b200.models import TransformerConfig
    from terapipe_b200.runtime.engine import StageEngine
    cfg = TransformerConfig(batch_size=3, seq_len=128, n_layers=2, embedding_dim=256,
                            num_attention_heads=4, n_devices=1)
    x = torch.randn(128, 3, 256, generator=torch.Generator().manual_seed(1))
    got = []
    for merged in (True, False):
        how = dict(use_graph=True) if merged else dict(use_graph=False, launch_plan=False)
        eng = StageEngine(cfg, batch_slices, seq_slices, loss_scale=1024.0, lr=1e-4, **how)
        assert eng._merged == merged
        eng.set_input(x)
        eng.compute_grads()
        grads = eng.named_grads()
        eng.grad.zero_()
        for _ in range(3):
            eng.step()
        eng.check_status()
        got.append((grads, eng.output().clone(), eng.master.clone(), eng.launch_count))
    for name, a in got[0][0].items():
        b = got[1][0][name]
        assert ((a - b).norm() / b.norm()).item() < 2e-3, name
    for a, b in zip(got[0][1:3], got[1][1:3]):
        assert ((a.float() - b.float()).norm() / b.float().norm()).item() < 2e-3
    assert got[0][3] <= got[1][3]
