"""Order of the sums in prompts over int8 and uint4 weights: uint4 rows have the bits of short calls, int8 rows over a copy of the codes those of
the kernel that expands the codes per tile."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from xfastertransformer_b200.runtime.loader import make_linear


def _weights(rows, K, kind, g):
    return make_linear(torch.randn(rows, K, generator=g, device="cuda") * 0.05, kind).to("cuda")


@pytest.mark.parametrize("T", [257, 400, 700])
@pytest.mark.parametrize("N_,K", [(264, 512), (1024, 488)])
def test_uint4_prompts_sum_as_short_calls(T, N_, K):
    """Reductions of up to four blocks of 128 have one part in any call."""
    from xfastertransformer_b200.ops import native as N
    g = torch.Generator(device="cuda").manual_seed(T + N_)
    x = torch.randn(T, K, generator=g, device="cuda").bfloat16()
    W, bias = _weights(N_, K, "int4", g), torch.randn(N_, generator=g, device="cuda")
    pieces = x.split(64)
    assert torch.equal(N.linear(x, W, bias, out_dtype=torch.float32), torch.cat([N.linear(p, W, bias, out_dtype=torch.float32) for p in pieces]))
    assert torch.equal(N.linear_gated(x, W), torch.cat([N.linear_gated(p, W) for p in pieces]))


@pytest.mark.parametrize("T,N_,K,gated", [(129, 136, 128, False), (200, 4096, 4096, False), (300, 19000, 1032, False), (700, 4104, 2048, False),
                                          (330, 640, 528, True), (700, 9600, 1024, True)])
@pytest.mark.parametrize("zero", [True, False])
def test_int8_prompts_give_one_set_of_bits(T, N_, K, gated, zero, monkeypatch):
    from xfastertransformer_b200.ops import native as N
    from xfastertransformer_b200.ops import native_quant as Q
    g = torch.Generator(device="cuda").manual_seed(T + N_)
    x = torch.randn(T, K, generator=g, device="cuda").bfloat16()
    rows = 2 * N_ if gated else N_
    W, bias = _weights(rows, K, "int8", g), torch.randn(rows, generator=g, device="cuda")
    res = torch.randn(T, N_, generator=g, device="cuda").bfloat16()
    if not zero:
        W.zero = None

    def both():
        if gated:
            return N.linear_gated(x, W, "silu", bias), N.linear_gated(x, W, "gelu")
        return N.linear(x, W, bias, None, res, 0.7, torch.float32), N.linear(x, W, bias, "gelu")

    got = both()
    monkeypatch.setattr(Q, "CODES_MAX_COPY", 0)
    assert all(torch.equal(a, b) for a, b in zip(got, both()))
