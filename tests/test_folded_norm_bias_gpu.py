"""Products with a folded norm and a bias (csrc/kernels/gemm_e4m3_sm100.cu): the sum times 1/rms is rounded to fp32 before the bias is added, so the
bias can be added behind the launch to the same bits.  A fused multiply-add in its place moves every logit of a model with QKV biases."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from xfastertransformer_b200.runtime.loader import make_linear


@pytest.mark.parametrize("T", [1, 8, 17, 32, 64])
@pytest.mark.parametrize("N_,K", [(1152, 896), (264, 1000), (4608, 3584)])
def test_bias_behind_the_rounded_product(T, N_, K):
    from xfastertransformer_b200.ops import native as N
    g = torch.Generator(device="cuda").manual_seed(T + N_ + K)
    x = torch.randn(T, K, generator=g, device="cuda").bfloat16()
    W = make_linear((torch.randn(N_, K, generator=g, device="cuda") * 0.03).bfloat16(), "bf16").to("cuda")
    bias = torch.randn(N_, generator=g, device="cuda")
    plain = N.linear_rms(x, W, 1e-6, out_dtype=torch.float32)
    got = N.linear_rms(x, W, 1e-6, bias, out_dtype=torch.float32)
    assert torch.equal(got, plain + bias)
    assert torch.equal(N.linear_rms(x, W, 1e-6, bias), (plain + bias).bfloat16())
