"""GeLU and its derivative in the GEMM epilogue, value by value against 64-bit arithmetic."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bn", [64, 1128, 1192, 1224, 1256])
def test_every_fp16_value(bn):
    """All finite fp16 values pass through an identity product.  The approximation's relative error
    (2e-6 with fp32 rounding of the exponent, up to |z| = 5.5 where fp16 ends) is far below the
    rounding of the result: half a unit in the last place, 2^-11 relative or 2^-25 absolute."""
    from terapipe_b200.ops import functional as F
    z = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(torch.float16)
    z = z[torch.isfinite(z)].view(-1, 256).cuda()
    eye = torch.eye(256, device="cuda", dtype=torch.float16)
    out, pre = torch.empty_like(z), torch.empty_like(z)
    F.gemm(z, eye, out, act="gelu", aux_out=pre, force_bn=bn)
    assert torch.equal(pre, z)
    zd = z.double()
    cdf = torch.special.erfc(-zd / math.sqrt(2)) / 2
    want = zd * cdf
    assert bool(((out.double() - want).abs() <= want.abs() * (2 ** -11 + 4e-6) + 2 ** -25 + 1e-9).all())
    d = torch.empty_like(z)
    F.gemm(torch.ones_like(z), eye, d, dact="gelu", aux_in=z, force_bn=bn)
    want = cdf + zd * torch.exp(-zd * zd / 2) / math.sqrt(2 * math.pi)
    assert bool(((d.double() - want).abs() <= want.abs() * 2 ** -11 + 2 ** -25 + 2e-6).all())
    F.check_device_status()


def test_infinities_and_nan_keep_to_themselves():
    from terapipe_b200.ops import functional as F
    x = torch.zeros(32, 64, device="cuda", dtype=torch.float16)
    w = torch.zeros(64, 64, device="cuda", dtype=torch.float16)
    bias = torch.zeros(64, device="cuda", dtype=torch.float16)
    bias[0], bias[3], bias[5] = math.inf, math.nan, -math.inf
    out, pre = torch.empty_like(x), torch.empty_like(x)
    F.gemm(x, w, out, bias=bias, act="gelu", aux_out=pre)
    assert bool((out[:, 0] == math.inf).all()) and bool(out[:, 3].isnan().all())
    assert bool((out[:, 5] == 0).all())
    rest = [j for j in range(64) if j not in (0, 3, 5)]
    assert bool((out[:, rest] == 0).all())
