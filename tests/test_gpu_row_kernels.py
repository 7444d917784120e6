"""The batched column sums and folds of a layer against fp64."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, ref):
    return ((a.double() - ref).norm() / ref.norm()).item()


@pytest.mark.parametrize("rows,widths", [(1, (8,)), (63, (264, 8)), (127, (256, 72)), (128, (512, 8, 1032, 256)),
                                         (1000, (768, 3072)), (4100, (2048, 512, 768, 1536))])
def test_layer_sums_and_folds(rows, widths):
    from terapipe_b200.ops.lib import check, cuda_lib
    g = torch.Generator(device="cuda").manual_seed(rows)
    n, H, parts = len(widths), 200, 37
    mats = [torch.randn(rows, w + 8, device="cuda", generator=g).half()[:, :w] for w in widths]
    db = [torch.randn(w, device="cuda", generator=g) for w in widths]
    slots = [torch.randn(parts, 2, H, device="cuda", generator=g) for _ in range(2)]
    dg, de = ([torch.randn(H, device="cuda", generator=g) for _ in range(2)] for _ in range(2))
    want = [b.double() + m.double().sum(0) for b, m in zip(db, mats)]
    want_g = [a.double() + s[:, 0].double().sum(0) for a, s in zip(dg, slots)]
    want_e = [a.double() + s[:, 1].double().sum(0) for a, s in zip(de, slots)]
    P = ctypes.c_void_p

    def ptrs(ts):
        return (P * len(ts))(*[t.data_ptr() for t in ts])

    check(cuda_lib().tp_layer_sums(0, n, ptrs(mats), (ctypes.c_longlong * n)(*[m.stride(0) for m in mats]),
                                   (ctypes.c_int * n)(*widths), ptrs(db), rows, 2, ptrs(slots), parts, H,
                                   ptrs(dg), ptrs(de), torch.cuda.current_stream().cuda_stream), "tp_layer_sums")
    for got, ref in zip(db + dg + de, want + want_g + want_e):
        assert _rel(got, ref) < 2e-6 * max(1.0, rows ** 0.5 / 8)   # fp32 sums of `rows` terms
    assert all(s.abs().max().item() == 0.0 for s in slots)
