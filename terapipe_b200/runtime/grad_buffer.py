"""Whether a stage's gradient buffer can hold anything but zeros."""
from __future__ import annotations

import torch


def _references(t: torch.Tensor) -> int:
    return torch._C._storage_Use_Count(t.untyped_storage()._cdata)


class GradBuffer:
    """``tensor`` is the owner's, which the library's kernels write through raw pointers; everybody else gets views of
    it (:meth:`share`).  An update leaves zeros, so that the next one need not look at the buffer, unless the owner
    left gradients in it (``left``) or somebody has, or has had, a view since then.  Torch's version counter
    cannot tell: writes of kernels and through ``.data`` leave it as it is, and tensors made under
    ``torch.inference_mode()`` have none."""

    def __init__(self, tensor: torch.Tensor):
        self.tensor = tensor
        self.left = False
        self._shared = False
        self._own = _references(tensor)

    def share(self) -> torch.Tensor:
        self._shared = True
        return self.tensor.detach()

    @property
    def may_hold(self) -> bool:
        return self.left or self._shared

    def cleared(self) -> None:
        """An update has left zeros.  Whoever still holds a view (or a view of one) may write at any time."""
        self.left = False
        if self._shared:
            self._shared = _references(self.tensor) > self._own
