"""Python entry points of the sm_100a kernels (torch tensors in, raw pointers out).

Every function enqueues on the current torch CUDA stream, allocates nothing unless the
caller omits an output/workspace tensor, and raises :class:`KernelError` when the native
call rejects its arguments.  Device-side wait time-outs are reported through a per-device
status word: call :func:`check_device_status` after a synchronisation point.
"""
from __future__ import annotations

import ctypes
from typing import Optional

import torch

from .lib import CHECK_CODES, _ERRORS, CheckFailed, CommTimeout, KernelError, check, cuda_lib

_ACT = {None: 0, "none": 0, "relu": 1, "gelu": 2}
_status = {}


_DT = {torch.float16: 0, torch.bfloat16: 1}


def _dt(t: torch.Tensor) -> int:
    code = _DT.get(t.dtype)
    if code is None:
        raise KernelError(f"unsupported dtype {t.dtype}; kernels take float16 or bfloat16")
    return code


def _ptr(t: Optional[torch.Tensor]) -> Optional[int]:
    return None if t is None else t.data_ptr()


# A short slice's layer is 14 calls of a few microseconds of device work each, so what a call costs here counts:
# 16 us for gemm() with torch.cuda.current_stream() (3.2, the object it makes) and a method call for every size and
# stride, 9 with the raw handle and one tuple each.
def _stream() -> int:
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def _status_ptr(t: torch.Tensor) -> int:
    word = _status.get(t.get_device())
    return (status_word(t.device) if word is None else word).data_ptr()


def status_word(device=None) -> torch.Tensor:
    """int32[1] on the device; kernels CAS their first time-out code into it."""
    idx = None if device is None else torch.device(device).index
    if idx is None:
        idx = torch.cuda.current_device()
    if idx not in _status:
        _status[idx] = torch.zeros(1, dtype=torch.int32, device=f"cuda:{idx}")
    return _status[idx]


def check_device_status(device=None, reset=True) -> None:
    """Synchronising read of the status word; raises :class:`CommTimeout` if a wait ran out and
    :class:`CheckFailed` if an index check of the checked build failed."""
    word = status_word(device)
    code = int(word.item())
    if code != 0:
        if reset:
            word.zero_()
        if code in CHECK_CODES:
            raise CheckFailed(f"{_ERRORS.get(code, 'checked build: index check failed')} (code {code})")
        raise CommTimeout(f"a device-side wait timed out (code {code})")


def gemm(a: torch.Tensor, b: torch.Tensor, out: torch.Tensor, *, a_mn=False, b_mn=False,
         alpha: float = 1.0, bias=None, residual=None, act=None, aux_out=None, dact=None,
         aux_in=None, accumulate=False, force_bn: int = 0) -> torch.Tensor:
    """``out[m, n] = epilogue(alpha * sum_k A(m, k) B(n, k))`` on tcgen05 tensor cores.

    ``a`` is ``[M, K]`` (or ``[K, M]`` when ``a_mn``), ``b`` is ``[N, K]`` (or ``[K, N]``
    when ``b_mn``); rows may be strided (last dim contiguous).  Epilogue options: ``bias``
    ``[N]``; ``act`` in {"relu", "gelu"} (``aux_out`` receives the pre-activation for
    gelu); ``residual`` ``[M, N]``; ``dact`` in {"relu", "gelu"} multiplies by the
    activation derivative evaluated on ``aux_in`` (post-activation for relu,
    pre-activation for gelu); ``out`` may be fp32 and may ``accumulate``."""
    M, N = out.shape
    rows, cols = a.shape, b.shape
    lda, ldb, ldo = a.stride(), b.stride(), out.stride()
    K = rows[0] if a_mn else rows[1]
    assert lda[-1] == 1 and ldb[-1] == 1 and ldo[-1] == 1
    assert (rows[1] if a_mn else rows[0]) == M, "A does not match out rows"
    assert (cols[1] if b_mn else cols[0]) == N and (cols[0] if b_mn else cols[1]) == K
    aux = aux_out if aux_out is not None else aux_in
    st = cuda_lib().tp_gemm(
        _dt(a), int(a_mn), int(b_mn), a.data_ptr(), lda[0], b.data_ptr(), ldb[0],
        out.data_ptr(), ldo[0], int(out.dtype == torch.float32), int(accumulate), M, N, K, float(alpha),
        None if bias is None else bias.data_ptr(), None if residual is None else residual.data_ptr(),
        0 if residual is None else residual.stride(0), _ACT[act], None if aux_out is None else aux_out.data_ptr(),
        _ACT[dact], None if aux_in is None else aux_in.data_ptr(), 0 if aux is None else aux.stride(0),
        int(force_bn), _status_ptr(a), _stream())
    if st:
        check(st, "tp_gemm")
    return out


GEMM_TRACE_SLOTS = 24


def gemm_pair_trace(a: torch.Tensor, b: torch.Tensor, out: torch.Tensor, bn: int = 256) -> torch.Tensor:
    """Run the CTA-pair GEMM (fp16, ``out = a @ b.T``) in its tracing build and return the
    per-CTA phase stamps, an int64 tensor ``[n_ctas, 24]`` of SM clock cycles (slot meanings
    are listed at ``tp_gemm_trace`` in ``csrc/gemm_sm100.cu``)."""
    M, N = out.shape
    K = a.shape[1]
    assert a.dtype == torch.float16 and b.dtype == torch.float16 and out.dtype == torch.float16
    tiles = ((M + 255) // 256) * ((N + bn - 1) // bn)
    sms = torch.cuda.get_device_properties(a.device).multi_processor_count
    n_ctas = 2 * min(tiles, sms // 2)
    trace = torch.zeros(n_ctas, GEMM_TRACE_SLOTS, dtype=torch.int64, device=a.device)
    st = cuda_lib().tp_gemm_trace(int(bn), a.data_ptr(), a.stride(0), b.data_ptr(), b.stride(0),
                                  out.data_ptr(), out.stride(0), M, N, K, trace.data_ptr(),
                                  _status_ptr(a), _stream())
    check(st, "tp_gemm_trace")
    return trace


def layernorm_fwd(x, gamma, beta, y, mean, rstd, eps=1e-5):
    rows, H = x.shape
    st = cuda_lib().tp_layernorm_fwd(_dt(x), x.data_ptr(), gamma.data_ptr(), beta.data_ptr(),
                                     y.data_ptr(), mean.data_ptr(), rstd.data_ptr(), rows, H,
                                     float(eps), _stream())
    check(st, "tp_layernorm_fwd")
    return y


def layernorm_bwd_scratch_floats(rows: int, H: int) -> int:
    return cuda_lib().tp_layernorm_bwd_parts(int(rows)) * 2 * H


def layernorm_bwd(dy, x, mean, rstd, gamma, dx, dgamma, dbeta, scratch, dres=None):
    """``dx = LN'(dy) (+ dres)``; ``dgamma``/``dbeta`` (fp32) are accumulated into.
    ``scratch`` is an fp32 workspace of :func:`layernorm_bwd_scratch_floats` elements."""
    rows, H = x.shape
    assert scratch.numel() >= layernorm_bwd_scratch_floats(rows, H)
    st = cuda_lib().tp_layernorm_bwd(_dt(x), dy.data_ptr(), x.data_ptr(), mean.data_ptr(),
                                     rstd.data_ptr(), gamma.data_ptr(), _ptr(dres), dx.data_ptr(),
                                     dgamma.data_ptr(), dbeta.data_ptr(), scratch.data_ptr(),
                                     rows, H, _stream())
    check(st, "tp_layernorm_bwd")
    return dx


def colsum(dy, db):
    """``db[n] += sum_rows dy[row, n]`` (bias gradient), fp32 accumulation."""
    rows, N = dy.shape
    st = cuda_lib().tp_colsum(_dt(dy), dy.data_ptr(), dy.stride(0), rows, N, db.data_ptr(), _stream())
    check(st, "tp_colsum")
    return db


def adam_tick(state, beta1=0.9, beta2=0.999):
    check(cuda_lib().tp_adam_tick(state.data_ptr(), beta1, beta2, _stream()), "tp_adam_tick")


def fused_adam(grad, master, m, v, model, state, lr, beta1=0.9, beta2=0.999, eps=1e-8,
               weight_decay=0.0, grad_scale=1.0):
    """One pass over flat buffers: unscale the fp32 gradient, update fp32 ``master``/``m``/``v``,
    rewrite the 16-bit ``model`` copy and zero ``grad``.  ``state`` is float32[3] =
    (step, 1-beta1^t, 1-beta2^t), advanced on the device by :func:`adam_tick`."""
    n = grad.numel()
    st = cuda_lib().tp_fused_adam(_dt(model), grad.data_ptr(), master.data_ptr(), m.data_ptr(),
                                  v.data_ptr(), model.data_ptr(), n, state.data_ptr(), lr, beta1,
                                  beta2, eps, weight_decay, grad_scale, _stream())
    check(st, "tp_fused_adam")


def _wgrad_args(dy, x, out):
    """``[layers, rows, width]`` operands and ``[layers, M, N]`` fp32 output (or one layer without the dimension).
    The kernel reads ``x`` as ``dy``'s type and stores fp32, whatever the tensors are: other types end here."""
    dtype = _dt(dy)
    if x.dtype != dy.dtype:
        raise KernelError(f"operands of one type: {dy.dtype} and {x.dtype}")
    if out.dtype != torch.float32:
        raise KernelError(f"weight gradients and their optimizer state are float32, not {out.dtype}")
    dy, x, out = (t if t.dim() == 3 else t.unsqueeze(0) for t in (dy, x, out))
    n, K, M = dy.shape
    N = x.shape[2]
    assert x.shape[:2] == (n, K) and out.shape == (n, M, N)
    assert dy.stride(2) == 1 and x.stride(2) == 1 and out.stride(2) == 1
    return (dtype, dy.data_ptr(), dy.stride(1), dy.stride(0), x.data_ptr(), x.stride(1), x.stride(0)), \
           (out.stride(1), out.stride(0), n, M, N, K)


def weight_grad(dy, x, out, accumulate=False):
    """``out[l] (+)= dy[l]^T @ x[l]`` (fp32) for every layer: the weight gradients of one kind of a stage."""
    operands, sizes = _wgrad_args(dy, x, out)
    st = cuda_lib().tp_wgrad(*operands, out.data_ptr(), *sizes, int(accumulate), 0, _status_ptr(dy),
                             _stream())
    check(st, "tp_wgrad")
    return out


def weight_grad_adam(dy, x, master, m, v, model, state, lr, beta1=0.9, beta2=0.999, eps=1e-8,
                     weight_decay=0.0, grad_scale=1.0):
    """:func:`weight_grad` and :func:`fused_adam` in one kernel: the gradients of the ``[layers, M, N]`` matrices
    ``master``/``m``/``v``/``model`` are not stored."""
    operands, sizes = _wgrad_args(dy, x, master)
    for t, dtype in ((m, torch.float32), (v, torch.float32), (model, dy.dtype)):
        if t.dtype != dtype:
            raise KernelError(f"moments are float32 and the model copy is the operands' type, not {t.dtype}")
        assert t.shape == master.shape and t.stride() == master.stride()
    st = cuda_lib().tp_wgrad_adam(*operands, master.data_ptr(), m.data_ptr(), v.data_ptr(), model.data_ptr(), *sizes,
                                  state.data_ptr(), lr, beta1, beta2, eps, weight_decay, grad_scale,
                                  0, _status_ptr(dy), _stream())
    check(st, "tp_wgrad_adam")


def fused_adam_ranges(grad, master, m, v, model, state, ranges, layers: int, layer_stride: int, lr,
                      beta1=0.9, beta2=0.999, eps=1e-8, weight_decay=0.0, grad_scale=1.0):
    """:func:`fused_adam` on the ranges ``[(begin, length), ...]`` of every layer of the flat buffers.  The ranges
    lie inside the buffers, and one layer's before the next one's."""
    if any(t.dtype != torch.float32 for t in (grad, master, m, v, state)):
        raise KernelError("gradients, optimizer state and step state are float32")
    if ranges and layers > 0:
        lo, hi = min(r[0] for r in ranges), max(r[0] + r[1] for r in ranges)
        end = hi + (layers - 1) * layer_stride
        if lo < 0 or end > min(t.numel() for t in (grad, master, m, v, model)) or (layers > 1 and layer_stride < hi - lo):
            raise KernelError(f"ranges [{lo}, {hi}) of {layers} layers, {layer_stride} apart, do not fit the buffers")
    LL = ctypes.c_longlong * len(ranges)
    st = cuda_lib().tp_fused_adam_ranges(_dt(model), grad.data_ptr(), master.data_ptr(), m.data_ptr(),
                                         v.data_ptr(), model.data_ptr(), len(ranges), LL(*[r[0] for r in ranges]),
                                         LL(*[r[1] for r in ranges]), layers, layer_stride, state.data_ptr(), lr,
                                         beta1, beta2, eps, weight_decay, grad_scale, _stream())
    check(st, "tp_fused_adam_ranges")


def fill(t, value: float):
    check(cuda_lib().tp_fill(_dt(t), t.data_ptr(), t.numel(), float(value), _stream()), "tp_fill")
    return t


def attn_fwd(qkv, b: int, h: int, D: int, t: int, c: int, o, lse2, scale: float = 0.0):
    """Slice-causal attention forward.

    ``qkv``: full-length projection buffer ``[L, b, h*3*D]`` (per head q,k,v interleaved);
    rows ``[0, c+t)`` are read, the slice's queries are rows ``[c, c+t)``.
    ``o``: ``[t*b, h*D]`` output of the slice (row = position*b + batch).
    ``lse2``: fp32 ``[b*h, L]`` base-2 log-sum-exp, written at positions ``[c, c+t)``.
    ``scale``: multiplier of q.k (0 = ``D ** -0.5``); heads narrower than ``D`` whose extra
    columns are zero pass the scale of their real width."""
    st = cuda_lib().tp_attn_fwd_scaled(_dt(qkv), D, float(scale), qkv.data_ptr(), b, h, t, c,
                                       o.data_ptr(), o.stride(0), lse2.data_ptr(), lse2.stride(0),
                                       _status_ptr(qkv), _stream())
    check(st, "tp_attn_fwd_scaled")
    return o


def attn_bwd(qkv, b: int, h: int, D: int, t: int, c: int, q_end: int, o, do_full, lse2, delta,
             dqkv, scale: float = 0.0):
    """Slice-causal attention backward for the slice ``[c, c+t)``.

    Slices are processed last to first.  ``do_full`` is the full-length gradient of the
    attention output ``[L*b, h*D]``: rows of the slices after this one (up to position
    ``q_end``) were written by their own backward, rows ``[c*b, (c+t)*b)`` by the caller just
    before this call.  ``o`` is this slice's forward output ``[t*b, h*D]``; ``lse2`` and
    ``delta`` are fp32 ``[b*h, L]`` (``delta`` rows of this slice are written here).
    Writes the slice's complete ``d(qkv)`` ``[t*b, h*3*D]``."""
    st = cuda_lib().tp_attn_bwd_scaled(_dt(qkv), D, float(scale), qkv.data_ptr(), b, h, t, c, q_end,
                                       o.data_ptr(), o.stride(0), do_full.data_ptr(),
                                       do_full.stride(0), lse2.data_ptr(), lse2.stride(0),
                                       delta.data_ptr(), dqkv.data_ptr(), dqkv.stride(0),
                                       _status_ptr(qkv), _stream())
    check(st, "tp_attn_bwd_scaled")
    return dqkv
