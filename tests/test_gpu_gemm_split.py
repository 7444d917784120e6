"""Products of few tiles: tiles of 32 columns, and K shared by the CTAs of a cluster."""
import pytest
import torch

pytestmark = pytest.mark.gpu

CODES = [32] + [parts * 10000 + bn for bn in (64, 128) for parts in (1, 2, 4, 8)]


def _gelu_grad(z):
    z = z.requires_grad_()
    return torch.autograd.grad(torch.nn.functional.gelu(z).sum(), z)[0].detach()


# rows below, at and past a tile (and of several), columns that end inside an owner's share, K of less than a stage,
# of an odd number of them and of many (the parts of K differ in length)
@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (77, 72, 1000), (8, 768, 3072), (128, 200, 136), (129, 136, 1160),
                                   (300, 456, 2056), (256, 64, 520)])
@pytest.mark.parametrize("b_mn", [False, True])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_every_split_and_epilogue(M, N, K, b_mn, dtype):
    from terapipe_b200.ops import functional as F
    gen = torch.Generator(device="cuda").manual_seed(M + N + K)

    def rand(*shape, scale=1.0):
        return (torch.randn(*shape, device="cuda", generator=gen) * scale).to(dtype)

    a, w = rand(M, K + 8)[:, :K], rand(*((K, N) if b_mn else (N, K)), scale=K ** -0.5)
    bias, res, pre = rand(N), rand(M, N), rand(M, N)
    plain = a.double() @ (w.double() if b_mn else w.double().t())
    z = plain + bias.double()
    gelu = torch.nn.functional.gelu
    eps = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    cases = [(dict(), plain), (dict(bias=bias, residual=res, alpha=0.5), 0.5 * plain + bias.double() + res.double()),
             (dict(bias=bias, act="relu"), z.relu()), (dict(bias=bias, act="gelu"), gelu(z)),
             (dict(dact="relu", aux_in=pre), plain * (pre.double() > 0)),
             (dict(dact="gelu", aux_in=pre), plain * _gelu_grad(pre.double()))]
    for code in CODES:
        if (K + 127) // 128 < code // 10000:
            continue
        for kw, want in cases:
            wide = torch.full((M, N + 16), float("nan"), device="cuda", dtype=dtype)
            out = wide[:, 8:N + 8]
            aux = torch.full((M, N), float("nan"), device="cuda", dtype=dtype) if kw.get("act") == "gelu" else None
            F.gemm(a, w, out, b_mn=b_mn, force_bn=code, aux_out=aux, **kw)
            # one rounding of the result (of values of magnitude 1) and fp32 sums of K products
            assert (out.double() - want).abs().max().item() < 2 * eps * (1 + want.abs().max().item()), (code, kw.keys())
            assert wide[:, :8].isnan().all() and wide[:, -8:].isnan().all()
            if aux is not None:
                assert (aux.double() - z).abs().max().item() < 2 * eps * (1 + z.abs().max().item())
            again = torch.empty(M, N, device="cuda", dtype=dtype)
            F.gemm(a, w, again, b_mn=b_mn, force_bn=code, **kw)
            assert torch.equal(again, out)
    F.check_device_status()


def test_refused_splits():
    from terapipe_b200.ops import functional as F
    from terapipe_b200.ops.lib import KernelError
    a, w = torch.randn(64, 512, device="cuda").half(), torch.randn(64, 512, device="cuda").half()
    for code, out in ((30064, torch.empty(64, 64, device="cuda").half()), (80064, torch.empty(64, 64, device="cuda").half()),
                      (160064, torch.empty(64, 64, device="cuda").half()), (20256, torch.empty(64, 64, device="cuda").half()),
                      (20064, torch.empty(64, 64, device="cuda"))):
        with pytest.raises(KernelError):
            F.gemm(a, w, out, force_bn=code)


@pytest.mark.parametrize("M,N,K,b_mn", [(77, 768, 3072, False), (256, 2048, 8192, True), (16, 8192, 2048, False),
                                        (128, 1024, 4096, True)])
def test_ordinary_calls_split(M, N, K, b_mn):
    """The choice's own codes, against the same product on a one-CTA tile."""
    from terapipe_b200.ops import functional as F
    from terapipe_b200.ops.lib import host_lib
    assert host_lib().tp_choose_small(M, N, K, int(b_mn), 0, 148) >= 20000
    torch.manual_seed(1)
    a = torch.randn(M, K, device="cuda").half()
    w = (torch.randn(*((K, N) if b_mn else (N, K)), device="cuda") * K ** -0.5).half()
    out = [torch.empty(M, N, device="cuda").half() for _ in range(2)]
    F.gemm(a, w, out[0], b_mn=b_mn)
    F.gemm(a, w, out[1], b_mn=b_mn, force_bn=128)
    F.check_device_status()
    # the same sums in another order, rounded to 11 bits
    assert ((out[0] - out[1]).float().abs() <= 2.0 ** -10 * (0.25 + out[1].float().abs())).all()
