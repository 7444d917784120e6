"""Both forms of the epilogue (operands asked for ahead of their chunk, and at its start) where the choice between them lies."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _grad(z):
    z = z.requires_grad_()
    return torch.autograd.grad(torch.nn.functional.gelu(z).sum(), z)[0].detach()


def _check(M, N, K, code, dtype, rows_apart):
    """`rows_apart` 0: one row for all, which no tensor map describes."""
    from terapipe_b200.ops import functional as F
    gen = torch.Generator(device="cuda").manual_seed(M + N + K)

    def rand(*shape, scale=1.0):
        return (torch.randn(*shape, device="cuda", generator=gen) * scale).to(dtype)

    def mat():
        return rand(M, N) if rows_apart else rand(1, N).expand(M, N)

    a, w, bias, res, aux = rand(M, K), rand(N, K, scale=K ** -0.5), rand(N), mat(), mat()
    plain = a.double() @ w.double().t()
    eps = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    z = plain + bias.double()
    for kw, want in ((dict(bias=bias), z), (dict(bias=bias, act="gelu"), torch.nn.functional.gelu(z)),
                     (dict(bias=bias, residual=res), z + res.double()),
                     (dict(dact="gelu", aux_in=aux), plain * _grad(aux.double())),
                     (dict(dact="relu", aux_in=aux, residual=res), (plain + res.double()) * (aux.double() > 0))):
        wide = torch.full((M, N + 16), float("nan"), device="cuda", dtype=dtype)
        F.gemm(a, w, wide[:, 8:N + 8], force_bn=code, **kw)
        # one rounding of the result (of values of magnitude 1) and fp32 sums of K products
        assert (wide[:, 8:N + 8].double() - want).abs().max().item() < 2 * eps * (1 + want.abs().max().item()), kw.keys()
        assert wide[:, :8].isnan().all() and wide[:, -8:].isnan().all()
    F.check_device_status()


# several tiles a CTA with a short K (at the start of a chunk) and a long one (ahead), one tile a CTA
@pytest.mark.parametrize("M,N,K", [(300, 20008, 72), (1030, 10248, 4096), (130, 1544, 200)])
@pytest.mark.parametrize("code", (32, 64, 128, 256, 512, 1128, 1256))
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_forms(M, N, K, code, dtype):
    _check(M, N, K, code, dtype, rows_apart=True)


@pytest.mark.parametrize("M,N,K", [(1, 72, 136), (257, 264, 136), (9000, 776, 64), (300, 1000, 4104)])
@pytest.mark.parametrize("code", (0, 32, 64, 256, 1128, 1192, 40064))
def test_one_row_for_all(M, N, K, code):
    if code >= 20000 and K < 512:
        code = 10064
    _check(M, N, K, code, torch.float16, rows_apart=False)
