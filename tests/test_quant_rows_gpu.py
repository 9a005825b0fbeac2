"""Rows on their way into 8-bit products (csrc/kernels/quant_rows.cu): a norm in the same launch gives the bits of the norm and the codes
apart, at the sizes between which it runs, and rows of every kernel size hold what they stand for."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from xfastertransformer_b200.runtime.loader import make_linear


@pytest.mark.parametrize("K", [2048, 2056, 4096, 4104, 8192])
@pytest.mark.parametrize("T", [1, 33])
def test_norm_in_the_same_launch(T, K):
    from xfastertransformer_b200.ops import native as N
    from xfastertransformer_b200.ops import native_quant as Q
    g = torch.Generator(device="cuda").manual_seed(T + K)
    x = torch.randn(T, K, generator=g, device="cuda").bfloat16() * 3
    gain = torch.rand(K, generator=g, device="cuda") + 0.5
    h = N.rmsnorm(x, gain, 1e-5)
    for got, want in ((Q.quant_act(x, K, (gain, 1e-5)), Q.quant_act(h, K)),
                      (Q.split_e4m3(x, K, True, True, norm=(gain, 1e-5)), Q.split_e4m3(h, K, True, True)),
                      (Q.split_e4m3(x, K, norm=(gain, 1e-5))[:2], Q.split_e4m3(h, K)[:2])):
        assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("kind,N_", [("w8a8", 264), ("int4", 264), ("fp8", 256), ("fp8", 264), ("int8", 264)])
@pytest.mark.parametrize("T,K", [(5, 1024), (5, 2048), (70, 4096), (400, 4096), (3, 8208)])
@pytest.mark.parametrize("gated", [False, True])
def test_products_of_normalised_rows(kind, N_, T, K, gated):
    """norm_linear against its two steps, inside and outside of the sizes that one launch takes."""
    from xfastertransformer_b200.ops import native as N
    g = torch.Generator(device="cuda").manual_seed(T + K)
    x = torch.randn(T, K, generator=g, device="cuda").bfloat16()
    gain = torch.rand(K, generator=g, device="cuda") + 0.5
    W = make_linear(torch.randn(2 * N_ if gated else N_, K, generator=g, device="cuda") * 0.05, kind).to("cuda")
    h = N.rmsnorm(x, gain, 1e-5)
    want = N.linear_gated(h, W, "silu") if gated else N.linear(h, W)
    assert torch.equal(N.norm_linear(x, gain, 1e-5, W, None, "silu" if gated else None, gated), want)


@pytest.mark.parametrize("K", [8, 200, 4096, 4128, 8200, 16392, 32768, 32800])
def test_codes_of_every_row_length(K):
    from xfastertransformer_b200.ops import native_quant as Q
    g = torch.Generator(device="cuda").manual_seed(K)
    x = torch.randn(3, K, generator=g, device="cuda").bfloat16()
    q, s, z, n = Q.quant_act(x, K)
    assert torch.equal(n, q.float().sum(1))
    assert bool(((q.double() * s.double()[:, None] + z.double()[:, None] - x.double()).abs() <= 0.5001 * s.double()[:, None]).all())
    xs, st, sm = Q.split_e4m3(x, K, False, True)
    half = xs.shape[1] // 2
    back = (xs[:, :half].view(torch.float8_e4m3fn).double() + xs[:, half:].view(torch.float8_e4m3fn).double() / 16) * st.double()[:, None]
    top = x.double().abs().amax(1, keepdim=True)
    assert bool(((back[:, :K] - x.double()).abs() <= 2.0 ** -21 * top).all()) and bool((back[:, K:] == 0).all())
    assert bool(((sm.double() - x.double().sum(1)).abs() <= 2.0 ** -20 * x.double().abs().sum(1)).all())
