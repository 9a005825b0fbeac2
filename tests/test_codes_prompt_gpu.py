"""Prompts over int8 and uint4 weights through a copy of the codes in bf16 (csrc/kernels/gemm_prefill_sm100.cu): the line above which that
runs, ragged rows, features and reductions, bias, residual and fp32 rows, gated forms, weights without zero points."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from xfastertransformer_b200.ops import reference as R
from xfastertransformer_b200.runtime.loader import make_linear


@pytest.mark.parametrize("kind", ["int8", "int4"])
@pytest.mark.parametrize("T,N,K", [(129, 136, 8), (257, 1000, 200), (321, 264, 1032), (513, 4104, 528), (700, 256, 4120)])
def test_matches_64_bits(kind, T, N, K):
    """fp32 outputs: the codes are exact in bf16, so only the fp32 sums of n <= 2^13 products round (the codes and the zero point apart,
    each several times the weight)."""
    from xfastertransformer_b200.ops import native as Nat
    g = torch.Generator(device="cuda").manual_seed(T + N + K)
    x = torch.randn(T, K, generator=g, device="cuda").bfloat16()
    W = make_linear(torch.randn(N, K, generator=g, device="cuda") * 0.05, kind).to("cuda")
    bias, res = torch.randn(N, generator=g, device="cuda"), torch.randn(T, N, generator=g, device="cuda").bfloat16()
    got = Nat.linear(x, W, bias, None, res, 0.5, out_dtype=torch.float32)
    rows = Nat.linear(x, W, bias, "gelu", res, 0.5)
    Nat.Workspace.get(x.device).check_status()
    w = R.dequant_weight(W).double()
    y = x.double() @ w.t() + bias.double()
    mag = x.double().abs() @ (w.abs().t() + W.zero.double().abs()[None] * 2) + bias.double().abs() + res.double().abs()
    assert bool(((got.double() - y - 0.5 * res.double()).abs() <= 2.0 ** -18 * mag).all())
    want = torch.nn.functional.gelu(y, approximate="tanh") + 0.5 * res.double()
    assert bool(((rows.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -17 * mag + 2.0 ** -10).all())


@pytest.mark.parametrize("kind", ["int8", "int4"])
@pytest.mark.parametrize("T,I,K", [(330, 640, 528), (400, 136, 1032), (700, 1024, 1024)])
@pytest.mark.parametrize("zero", [True, False])
def test_gated_matches_its_parts(kind, T, I, K, zero):
    from xfastertransformer_b200.ops import native as Nat
    g = torch.Generator(device="cuda").manual_seed(T + I)
    x = torch.randn(T, K, generator=g, device="cuda").bfloat16()
    W = make_linear(torch.randn(2 * I, K, generator=g, device="cuda") * 0.05, kind).to("cuda")
    if not zero:
        W.zero = None
    gu = Nat.linear(x, W, out_dtype=torch.float32).double()
    want = torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]
    got = Nat.linear_gated(x, W, "silu").double()
    Nat.Workspace.get(x.device).check_status()
    assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -16 * gu.abs().amax()).all())


def test_without_room_for_the_copy(monkeypatch):
    """Where the copy has no room the kernels that expand per tile take the product, as they did all of them."""
    from xfastertransformer_b200.ops import native as Nat
    from xfastertransformer_b200.ops import native_quant as Q
    x = torch.randn(400, 512, device="cuda").bfloat16()
    W = make_linear(torch.randn(256, 512, device="cuda") * 0.05, "int4").to("cuda")
    want = Nat.linear(x, W, out_dtype=torch.float32)
    monkeypatch.setattr(Q, "CODES_MAX_COPY", 0)
    got = Nat.linear(x, W, out_dtype=torch.float32)
    assert bool(((got - want).abs() <= 2.0 ** -14 * want.abs().amax()).all())
