"""LayerNorm at every geometry of its kernels (warps per row, vectors per lane, rows that leave row
groups empty) and the batched column sums, against fp64."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, ref):
    return ((a.double() - ref).norm() / ref.norm()).item()


# (csrc/ln_geometry.h) H: 1, 2, 4, 8 and 16 warps a row, columns that end inside a vector round; rows: one, fewer than
# and just more than a CTA holds, more than one round of all CTAs
@pytest.mark.parametrize("H,rows", [(8, 5), (264, 25), (1024, 3700), (1600, 13), (2048, 1800), (2560, 7),
                                    (4096, 900), (5120, 500), (8200, 3), (12288, 160),
                                    # one round of one, two and four vectors a lane; 24 warps of four
                                    (768, 40), (2304, 300), (5120, 64), (1600, 1100), (4096, 590), (8192, 2049),
                                    (16384, 160)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_layernorm_geometries(H, rows, dtype):
    from terapipe_b200.ops import functional as F
    g = torch.Generator(device="cuda").manual_seed(H + rows)
    x, dy, dres = (torch.randn(rows, H, device="cuda", generator=g).to(dtype) for _ in range(3))
    gamma = (1 + 0.1 * torch.randn(H, device="cuda", generator=g)).to(dtype)
    beta = (0.1 * torch.randn(H, device="cuda", generator=g)).to(dtype)
    y, dx = torch.empty_like(x), torch.empty_like(x)
    mean, rstd = torch.empty(rows, device="cuda"), torch.empty(rows, device="cuda")
    F.layernorm_fwd(x, gamma, beta, y, mean, rstd)
    dgamma, dbeta = torch.ones(H, device="cuda"), torch.full((H,), 2.0, device="cuda")
    scratch = torch.full((F.layernorm_bwd_scratch_floats(rows, H),), float("nan"), device="cuda")
    F.layernorm_bwd(dy, x, mean, rstd, gamma, dx, dgamma, dbeta, scratch, dres=dres)
    x64, ga, be = (t.double().requires_grad_() for t in (x, gamma, beta))
    ref = torch.nn.functional.layer_norm(x64, (H,), ga, be)
    ref.backward(dy.double())
    eps = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8    # rounding of the 16-bit results
    assert _rel(y, ref.detach()) < eps and _rel(dx, x64.grad + dres.double()) < eps
    # fp32 sums over the rows of values computed in fp32
    assert _rel(dgamma, ga.grad + 1) < 2e-5 and _rel(dbeta, be.grad + 2) < 2e-5


@pytest.mark.parametrize("rows,widths", [(1, (8,)), (63, (264, 8)), (127, (256, 72)), (128, (512, 8, 1032, 256)),
                                         (1000, (768, 3072)), (4100, (2048, 512, 768, 1536)), (70, (32768,)),
                                         (1025, (12288, 16384, 4096)),
                                         # 256-column blocks: 48 of them in 8 chunks, 200 in 2, 320 in 4
                                         (2100, (12288,)), (1100, (10240, 40960)), (1030, (81920,))])
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
