"""When a gradient buffer may hold something that torch has not counted as a write."""
import pytest
import torch

from terapipe_b200.runtime.grad_buffer import GradBuffer


@pytest.mark.parametrize("inference", [False, True])
def test_views_handed_out_and_held(inference):
    with torch.inference_mode(inference):
        g = GradBuffer(torch.zeros(64))
        assert not g.may_hold
        g.share().data.add_(1.0)                 # (a write that leaves the version counter as it is)
        assert g.may_hold and g.tensor.sum() == 64
        g.cleared()
        assert not g.may_hold                    # nobody has a view any more
        part = g.share()[8:16].view(2, 4).data
        for _ in range(2):
            g.cleared()
            assert g.may_hold                    # a view of a view is held
        part.fill_(2.0)
        assert g.tensor.sum() == 56 + 16
        del part
        g.cleared()
        assert not g.may_hold
        g.left = True
        assert g.may_hold
        g.cleared()
        assert not g.may_hold
