"""The tiles of the token-major prompt product: which one a shape gets, and each of them at partial token blocks, feature
tiles that are not full and short or ragged reductions."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _bound(want, mag):
    """bf16 output (half a unit is 2^-9 of the value) of sums whose rounding is far below 2^-18 of the sum of magnitudes."""
    return 2.0 ** -8 * want.abs() + 2.0 ** -18 * mag + 1e-30


# 256 x 256 pairs (plain, gated), 256 x 128 pairs (plain, gated), 128 x 128 (plain, gated), rows that 32-byte stores do not fit
@pytest.mark.parametrize("T,N,K,gated", [(2300, 8184, 4096, False), (1500, 6000, 4096, True), (500, 4096, 11000, False),
                                         (160, 4096, 8192, True), (140, 136, 64, False), (385, 72, 200, True),
                                         (257, 8, 8, False), (129, 1000, 1032, False)])
def test_tiles_match_fp32(T, N, K, gated):
    from xfastertransformer_b200.ops import native as N_
    g = torch.Generator(device="cuda").manual_seed(T + N + K)
    x = torch.randn(T, K, generator=g, device="cuda").bfloat16()
    w = (torch.randn(2 * N if gated else N, K, generator=g, device="cuda") * 0.05).bfloat16()
    res = None if gated else torch.randn(T, N, generator=g, device="cuda").bfloat16()
    y, mag = x.double() @ w.double().t(), x.abs().double() @ w.abs().double().t()
    if gated:
        s = torch.nn.functional.silu(y[:, :N])
        want = s * y[:, N:]
        mag = 1.1 * mag[:, :N] * y[:, N:].abs() + s.abs() * mag[:, N:] + want.abs()
    else:
        want = y + res.double()
    got = N_.gemm_bf16(x, w, N, gated=gated, dual_off=N if gated else 0, act="silu" if gated else None, residual=res)
    N_.Workspace.get(x.device).check_status()
    err = (got.double() - want).abs()
    assert bool((err <= _bound(want, mag)).all()), (err / _bound(want, mag)).max().item()


@pytest.mark.parametrize("T,E,k,I,H", [(1100, 4, 2, 264, 512), (1024, 2, 1, 128, 136), (1290, 5, 2, 72, 256)])
def test_expert_tiles_of_256_rows(T, E, k, I, H):
    """At least 512 rows per expert on average: pairs of CTAs; uneven loads, an expert without tokens, tiles cut at 1..255 rows."""
    from xfastertransformer_b200.ops import native as N_
    from xfastertransformer_b200.ops import native_moe
    from xfastertransformer_b200.runtime.loader import make_linear
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, H, generator=g, device="cuda").bfloat16()
    ws = [(torch.randn(2 * I, H, generator=g, device="cuda") * 0.1, torch.randn(H, I, generator=g, device="cuda") * 0.1) for _ in range(E)]
    experts = [(make_linear(a.bfloat16(), "bf16"), make_linear(b.bfloat16(), "bf16")) for a, b in ws]
    idx = torch.rand(T, E - (E > 2), generator=g, device="cuda").topk(k, 1)[1].int()        # the last expert of E > 2 is empty
    wt = torch.rand(T, k, generator=g, device="cuda") + 0.1
    got = native_moe.moe_experts(x, idx, wt, experts)
    N_.Workspace.get(x.device).check_status()
    want = torch.zeros(T, H, dtype=torch.float64, device="cuda")
    tol = torch.zeros_like(want)
    for e, (a, b) in enumerate(experts):
        gu = x.double() @ a.w.double().t()
        h = torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]
        y = h @ b.w.double().t()
        s = ((idx == e) * wt).sum(1, keepdim=True).double()
        want += s * y
        # h and y are rounded to bf16 on the way
        tol += s * (2.0 ** -8 * y.abs() + 2.0 ** -8 * (h.abs() @ b.w.abs().double().t()))
    assert bool(((got.double() - want).abs() <= tol + 1e-5).all())
