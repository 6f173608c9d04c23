"""Forward GEMM at the edges of its tiles and of the rule that picks 128- or 256-column tiles (run on a B200)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(1, 256, 64), (127, 256, 128), (37889, 256, 256), (37889, 264, 256), (18945, 512, 72), (9473, 1024, 512),
                                   (9473, 1024, 8), (40000, 128, 256), (300, 40, 256)])
@pytest.mark.parametrize("act", [None, "relu"])
def test_forward_tiles(m, n, k, act):
    from gt_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn(m, k, generator=g, device="cuda").bfloat16()
    b = torch.randn(n, k, generator=g, device="cuda").bfloat16()
    bias = torch.randn(n, generator=g, device="cuda")
    got = native.gemm_nt(a, b, bias, act).double()
    want = a.double() @ b.double().t() + bias.double()
    want = want.relu() if act else want
    # bf16 result: half an ulp is 2^-9 of the value; fp32 accumulation of k exact products: k * 2^-24 of the sum of magnitudes
    bound = 2.0 ** -8 * want.abs() + k * 2.0 ** -23 * (a.double().abs() @ b.double().abs().t())
    assert bool(((got - want).abs() <= bound).all())
