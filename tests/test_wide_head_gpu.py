"""Wide products of 33 to 64 rows on the decode pipeline (csrc/kernels/gemm_e4m3_sm100.cu): more tiles than SMs, a last one cut short, and the
reductions between which the kernels change."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from xfastertransformer_b200.runtime.loader import make_linear


@pytest.mark.parametrize("T", [33, 64])
@pytest.mark.parametrize("N_,K", [(18952, 512), (18952, 520), (19100, 1032), (32000, 2048)])
def test_wide_products(T, N_, K):
    from xfastertransformer_b200.ops import native as N
    g = torch.Generator(device="cuda").manual_seed(T + N_ + K)
    x = torch.randn(T, K, generator=g, device="cuda").bfloat16()
    W = make_linear((torch.randn(N_, K, generator=g, device="cuda") * 0.02).bfloat16(), "bf16").to("cuda")
    bias = torch.randn(N_, generator=g, device="cuda")
    xd, wd = x.double(), W.w.double()
    r = torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-6)
    got = N.linear_rms(x, W, 1e-6, bias, out_dtype=torch.float32)
    N.Workspace.get(x.device).check_status()
    # fp32 sums of n <= 2^11 products: a few times 2^-24 sqrt(n) of the sum of magnitudes
    mag = (r * xd).abs() @ wd.t().abs() + bias.double().abs()
    assert bool(((got.double() - (r * xd) @ wd.t() - bias.double()).abs() <= 2.0 ** -18 * mag).all())
