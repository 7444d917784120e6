"""The matrices that a product's epilogue reads, as tiles and where no tensor map describes them."""
import pytest
import torch

pytestmark = pytest.mark.gpu

TILES = (32, 64, 128, 256, 512, 1128, 1192, 1224, 1256)


def _check(M, N, K, code, dtype, ld=None, shift=0):
    """Residual, derivative's argument, and both; `ld`, `shift`: row stride and first element of the matrices."""
    from terapipe_b200.ops import functional as F
    gen = torch.Generator(device="cuda").manual_seed(M + N + K)

    def rand(*shape, scale=1.0):
        return (torch.randn(*shape, device="cuda", generator=gen) * scale).to(dtype)

    def mat():
        return torch.as_strided(rand(M * (ld or N) + shift), (M, N), (ld or N, 1), shift)

    a, w, bias, res, aux = rand(M, K), rand(K, N, scale=K ** -0.5), rand(N), mat(), mat()
    plain = a.double() @ w.double()
    z = aux.double().requires_grad_()
    grad = torch.autograd.grad(torch.nn.functional.gelu(z).sum(), z)[0]
    eps = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    for kw, want in ((dict(residual=res), plain + res.double()),
                     (dict(residual=res, bias=bias), plain + bias.double() + res.double()),
                     (dict(dact="gelu", aux_in=aux), plain * grad),
                     (dict(dact="relu", aux_in=aux, bias=bias), (plain + bias.double()) * (aux.double() > 0)),
                     (dict(dact="relu", aux_in=aux, residual=res), (plain + res.double()) * (aux.double() > 0))):
        wide = torch.full((M, N + 16), float("nan"), device="cuda", dtype=dtype)
        F.gemm(a, w, wide[:, 8:N + 8], b_mn=True, force_bn=code, **kw)
        # one rounding of values of magnitude 1, fp32 sums of K products
        assert (wide[:, 8:N + 8].double() - want).abs().max().item() < 2 * eps * (1 + want.abs().max().item()), kw.keys()
        assert wide[:, :8].isnan().all() and wide[:, -8:].isnan().all()
    F.check_device_status()


# rows and columns that end inside a tile and a 32 x 32 chunk; one chunk, and several tiles a CTA (each of a warp's
# four buffers many times over)
@pytest.mark.parametrize("M,N,K", [(1, 8, 64), (257, 264, 136), (300, 1000, 64), (9000, 1544, 64)])
@pytest.mark.parametrize("code", TILES)
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_tiles(M, N, K, code, dtype):
    _check(M, N, K, code, dtype)


@pytest.mark.parametrize("code", (64, 1128))
@pytest.mark.parametrize("M,ld,shift", [(300, 280, 0), (1, 301, 0), (1, 264, 8), (70, 264, 8)])
def test_other_strides(M, ld, shift, code):
    """Rows further apart; one row with a stride that only it may have; matrices that start inside a buffer."""
    _check(M, 264, 136, code, torch.float16, ld=ld, shift=shift)
