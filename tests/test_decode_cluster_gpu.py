"""bf16 products of at most 64 rows (xft_gemm_bf16_cluster in csrc/kernels/gemm_e4m3_sm100.cu): token tiles and their edges, ragged
features and reductions, clusters along K, gated, folded norm, and the query / key / value product with its cache rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from xfastertransformer_b200.runtime.loader import make_linear

# token tiles of 16, 32 and 64; K of one partial block of 64, a partial last block, enough for 8 parts; one tile more than there are SMs
SHAPES = [(1, 128, 64), (16, 136, 8), (17, 384, 200), (32, 1000, 1032), (33, 200, 4096), (64, 264, 2056), (31, 18952, 72), (64, 18944, 136)]


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("fold", [False, True])
@pytest.mark.parametrize("T,N,K", SHAPES)
def test_cluster_products_match_64_bits(T, N, K, fold, gated):
    """fp32 outputs: bf16 products are exact in fp32 and n <= 2^12 of them add up with an error of a few times 2^-24 sqrt(n) of the sum
    of magnitudes; the norm's factor and the gate (slope at most 1.1) add a few roundings."""
    from xfastertransformer_b200.ops import native as Nat
    g = torch.Generator(device="cuda").manual_seed(T + N + K)
    x = torch.randn(T, K + 8, generator=g, device="cuda").bfloat16()[:, :K]                  # rows with a pitch
    rows = N * (1 + gated)
    w = (torch.randn(rows, K, generator=g, device="cuda") * 0.05).bfloat16()
    bias = torch.randn(rows, generator=g, device="cuda")
    res = None if fold or gated else torch.randn(T, N, generator=g, device="cuda").bfloat16()
    out = torch.empty(T, N, device="cuda")
    act, eps = "silu" if gated else None, 1e-5 if fold else None
    Nat._gemm_cluster(x, x.stride(0), w, out, T, N, K, gated, N if gated else 0, bias, res, N if res is not None else 0, 0.5, act, eps)
    Nat.Workspace.get(x.device).check_status()
    xd = x.double()
    if fold:
        xd = xd * torch.rsqrt(xd.pow(2).mean(1, keepdim=True) + eps)
    y = xd @ w.double().t() + bias.double()
    mag = xd.abs() @ w.double().abs().t() + bias.double().abs()
    want = torch.nn.functional.silu(y[:, :N]) * y[:, N:] if gated else y if res is None else y + 0.5 * res.double()
    tol = 2.0 ** -18 * mag
    tol = tol[:, :N] * (1.1 * y[:, N:].abs() + 1) + tol[:, N:] * (y[:, :N].abs() + 1) if gated else tol + (0 if res is None else 2.0 ** -22 * res.double().abs())
    assert bool(((out.double() - want).abs() <= tol).all()), ((out.double() - want).abs() / tol).max().item()


@pytest.mark.parametrize("fold", [False, True])
@pytest.mark.parametrize("T", [1, 4, 5, 16, 17, 32, 33, 64])
def test_qkv_in_one_and_two_launches_agree(T, fold, monkeypatch):
    """Both forms round q, k and v to bf16 before the rotation: a sum on the edge of a rounding differs by one step, twice 2^-8 of it."""
    from xfastertransformer_b200.ops import native as Nat
    hq, hkv, K = 6, 2, 328
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, K, generator=g, device="cuda").bfloat16()
    W = make_linear(torch.randn((hq + 2 * hkv) * 128, K, generator=g, device="cuda") * 0.05, "bf16").to("cuda")
    bias = torch.randn((hq + 2 * hkv) * 128, generator=g, device="cuda")
    table = torch.randn(80, 128, generator=g, device="cuda")
    pos = torch.arange(T, device="cuda").int()
    slots = torch.randperm(128, generator=g, device="cuda")[:T].int()
    qs = torch.rand(T, generator=g, device="cuda") + 0.5
    got = []
    for one in (True, False):
        monkeypatch.setattr(Nat, "_qkv_one_kernel", lambda *a: one)
        k, v = (torch.zeros(2, hkv, 64, 128, device="cuda").bfloat16() for _ in range(2))
        q = Nat.qkv_linear_rope_cache(x, W, bias, 1e-5 if fold else None, hq, hkv, pos, table, 128, "half", k, v, slots, qs)
        Nat.Workspace.get(x.device).check_status()
        got.append((q.float(), k.float(), v.float()))
    for a, b in zip(*got):
        assert bool(((a - b).abs() <= 2.0 ** -6 * a.abs().amax()).all()) and float((a - b).norm() / a.norm()) < 2.0 ** -9


@pytest.mark.parametrize("name,value", [("XFT_GEMM_STREAMK", "0"), ("XFT_GEMM_STREAMK", "2"), ("XFT_SK_CLUSTER", "4")])
def test_a_kernel_asked_for_by_name_is_taken(name, value, monkeypatch):
    from xfastertransformer_b200.ops import native as Nat
    from xfastertransformer_b200.utils.flags import Env
    assert Nat._use_cluster(16, 4096, 4096, False)
    try:
        monkeypatch.setenv(name, value)
        Env.get().reload()
        assert not Nat._use_cluster(16, 4096, 4096, False)
    finally:
        monkeypatch.undo()
        Env.get().reload()


@pytest.mark.parametrize("T", [16, 33, 64])
@pytest.mark.parametrize("N,K", [(12288, 4096), (4096, 4096), (896, 4864)])
def test_sums_are_no_further_off_than_those_of_the_older_kernels(T, N, K, monkeypatch):
    """fp32 results against 64 bits.  The sums of an accumulator are cut at its last bit, so their error grows with the k in it; a
    quarter of room for another order of the same sums."""
    from xfastertransformer_b200.ops import native as Nat
    g = torch.Generator(device="cuda").manual_seed(N + T)
    x = torch.randn(T, K, generator=g, device="cuda").bfloat16()
    W = make_linear(torch.randn(N, K, generator=g, device="cuda") * 0.02, "bf16").to("cuda")
    want = x.double() @ W.w.double().t()
    errors = []
    for use in (Nat._use_cluster, lambda *a: False):
        monkeypatch.setattr(Nat, "_use_cluster", use)
        errors.append(((Nat.linear(x, W, out_dtype=torch.float32).double() - want).norm() / want.norm()).item())
    Nat.Workspace.get(x.device).check_status()
    assert errors[0] <= 1.25 * errors[1], errors
