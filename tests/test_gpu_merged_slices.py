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
        eng = StageEngine(cfg, batch_slices, seq_slices, loss_scale=1024.0, lr=1e-4, use_graph=merged,
                          merge_slices=merged)
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


def _engine(**kw):
    from terapipe_b200.models import TransformerConfig
    from terapipe_b200.runtime.engine import StageEngine
    cfg = TransformerConfig(batch_size=2, seq_len=64, n_layers=1, embedding_dim=256,
                            num_attention_heads=4, n_devices=1)
    return StageEngine(cfg, [2], [24, 40], use_graph=False, **kw)


def test_refusing_plans_and_segment_graphs_leaves_the_schedule_alone():
    assert _engine()._merged
    assert _engine(launch_plan=False)._merged and _engine(segment_graphs=False)._merged
    assert not _engine(launch_plan=True)._merged and not _engine(segment_graphs=True)._merged
    assert not _engine(merge_slices=False)._merged


def test_trainer_takes_the_schedule():
    from terapipe_b200.runtime.trainer import Trainer
    for merge in (None, True, False):
        tr = Trainer("test", batch_size=2, n_layers=1, batch_slices=[2], seq_slices=[64, 64], merge_slices=merge)
        assert tr.engine._merged == (merge is not False)


def test_launches_are_those_of_the_pass_that_ran():
    """Counted by the calls into the library: one layer, two token slices."""
    from terapipe_b200.utils.trace import SliceTimeline
    eng = _engine(segment_graphs=False)
    lib, calls = eng.lib, []

    class Counting:
        def __getattr__(self, name):
            fn = getattr(lib, name)

            def call(*args):
                # attention's backward is three kernels in one call
                calls.append(3 if name.startswith("tp_attn_bwd") else 1)
                return fn(*args)
            return call

    eng.lib = Counting()
    for timeline in (None, SliceTimeline(stage=0), None):
        eng.timeline = timeline
        eng.set_input(torch.randn(64, 2, 256))
        before = eng.launch_count
        calls.clear()
        eng.step()
        # (the optimizer's two launches do not go through eng.lib)
        assert eng.launch_count - before == sum(calls) + 2
        assert sum(calls) == (12 + 4 + 5 if timeline is None else 2 * 16 + 5)


def _count_slices(monkeypatch):
    from terapipe_b200.runtime.engine import StageEngine
    seen, real = [], StageEngine._forward_slice
    monkeypatch.setattr(StageEngine, "_forward_slice", lambda self, sl: (seen.append(sl[3]), real(self, sl))[1])
    return seen


def test_runner_verify_runs_the_slices(monkeypatch):
    from terapipe_b200.models import TransformerConfig
    from terapipe_b200.runtime.runner import NCCLTransformerRunner
    cfg = TransformerConfig(batch_size=2, seq_len=64, n_layers=1, embedding_dim=256,
                            num_attention_heads=4, n_devices=1)
    runner = NCCLTransformerRunner(cfg, [2], [24, 40], "env://", 1, 1, 1, 1, 0, 0, mixed_precision=True)
    assert runner.merges_slices
    seen = _count_slices(monkeypatch)
    runner.verify()
    assert seen == [24, 40, 64]        # the sliced engine, then the whole sequence


def test_golden_check_runs_the_slices(monkeypatch, tmp_path):
    from terapipe_b200.runtime import verify
    kw = dict(model="test", n_layers=1, batch_size=2, device="cuda", engine="b200", dtype=torch.float16)
    verify.verify_one_step(str(tmp_path), "save", **kw)
    seen = _count_slices(monkeypatch)
    verify.verify_one_step(str(tmp_path), "load", n_input_slices=4, **kw)
    assert seen == [32] * 4


def test_a_turned_round_host_input_is_not_rearranged_on_the_host():
    """[B, L, H] in pinned memory, handed over as an [L, B, H] view."""
    from torch.utils._python_dispatch import TorchDispatchMode
    eng = _engine()
    x = torch.randn(2, 64, 256).half().pin_memory().transpose(0, 1)
    assert not x.is_contiguous()
    uploads = []

    class Watch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            if func is torch.ops.aten.copy_.default and not args[1].is_cuda and args[0].is_cuda:
                uploads.append(args[1].stride() == args[0].stride())
            return func(*args, **(kwargs or {}))

    with Watch():
        eng.set_input(x)
    assert all(uploads)
    assert torch.equal(eng.X[0].view(64, 2, 256).cpu(), x)


@pytest.mark.parametrize("failures", [0, 1, 2])
def test_capture_makes_room_when_memory_is_short(failures, monkeypatch):
    """Torch cannot give cached memory back while a capture runs: one that fails is tried again with
    the cache emptied, and a second failure leaves the step to smaller graphs."""
    import warnings
    from terapipe_b200.models import TransformerConfig
    from terapipe_b200.runtime.engine import StageEngine
    cfg = TransformerConfig(batch_size=2, seq_len=64, n_layers=1, embedding_dim=256,
                            num_attention_heads=4, n_devices=1)
    eng = StageEngine(cfg, [2], [64], use_graph=True, lr=1e-3)
    real, emptied, left = eng._iteration, [], [failures]

    def iteration(*args, **kw):
        real(*args, **kw)
        if torch.cuda.is_current_stream_capturing() and left[0]:
            left[0] -= 1
            raise torch.OutOfMemoryError("out of memory")

    monkeypatch.setattr(eng, "_iteration", iteration)
    monkeypatch.setattr(torch.cuda, "empty_cache",
                        lambda: emptied.append(torch.cuda.is_current_stream_capturing()))
    eng.set_input(torch.randn(64, 2, 256))
    with warnings.catch_warnings(record=True) as caught:
        warnings.simplefilter("always")
        for _ in range(3):
            eng.step()
    eng.check_status()
    assert (eng._graph is not None) == (failures < 2) and len(caught) == (failures == 2)
    assert emptied == [False] * (failures > 0)
    assert abs(eng.adam_state[0].item() - 3.0) < 1e-6 and eng.grad.abs().max().item() == 0.0
