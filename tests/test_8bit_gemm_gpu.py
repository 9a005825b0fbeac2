"""Products on the 8-bit tensor paths (csrc/kernels/gemm_e4m3_sm100.cu, W8A8 prompts in gemm_prefill_sm100.cu): token tiles and
their edges, ragged features and reductions, clusters along K, gated forms, rows of extreme range, experts by group."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from xfastertransformer_b200.ops import reference as R
from xfastertransformer_b200.runtime.loader import make_linear

# token tiles of 16, 32 and 64 and one past them; K of one partial block of 128, a partial last block, enough for 2 and 8 parts
SHAPES = [(1, 128, 128), (16, 136, 8), (17, 384, 200), (32, 1000, 1032), (33, 200, 4096), (64, 264, 2056), (65, 512, 1152), (200, 4096, 520)]


def _linear(w, kind):
    return make_linear(w, kind).to("cuda")


@pytest.mark.parametrize("kind", ["int4", "fp8"])
@pytest.mark.parametrize("T,N,K", SHAPES)
def test_split_activations_match_64_bits(kind, T, N, K):
    """fp32 outputs.  An activation is exact down to 2^-13 of its row's maximum and off by at most 2^-21 of it below; the fp32 sums of
    n <= 2^13 products may be off by a few times 2^-24 sqrt(n) of the sum of magnitudes."""
    from xfastertransformer_b200.ops import native as Nat
    g = torch.Generator(device="cuda").manual_seed(T + N + K)
    x = torch.randn(T, K, generator=g, device="cuda").bfloat16()
    x[0] *= 1e-30                                          # scales at both ends
    x[-1] = (x[-1].float() * torch.exp(4 * torch.randn(K, generator=g, device="cuda"))).bfloat16()      # long tails
    if T > 2:
        x[1], x[2] = 0, x[2] * 1e30
    W = _linear(torch.randn(N, K, generator=g, device="cuda") * 0.05, kind)
    bias, res = torch.randn(N, generator=g, device="cuda"), torch.randn(T, N, generator=g, device="cuda").bfloat16()
    got = Nat.linear(x, W, bias, None, res, 0.5, out_dtype=torch.float32)
    Nat.Workspace.get(x.device).check_status()
    w = R.dequant_weight(W).double()
    want = x.double() @ w.t() + bias.double() + 0.5 * res.double()
    # (uint4: codes and zero point are summed apart, each several times the weight)
    mag = x.double().abs() @ (w.abs().t() + (W.zero.double().abs()[None] * 2 if kind == "int4" else 0)) + bias.double().abs() + res.double().abs()
    low = x.double().abs().amax(1, keepdim=True) * w.abs().sum(1)[None]
    tol = 2.0 ** -18 * mag + 2.0 ** -21 * low
    assert bool(((got.double() - want).abs() <= tol).all()), ((got.double() - want).abs() / tol).max().item()


@pytest.mark.parametrize("kind", ["int4", "fp8", "w8a8"])
@pytest.mark.parametrize("T,I,K", [(3, 128, 256), (31, 384, 4112), (64, 256, 1040), (130, 640, 528), (700, 1024, 1024)])
def test_gated_matches_its_parts(kind, T, I, K):
    """act(gate) * up of one launch against the two products apart (fp32; W8A8 rounds gate and up to bf16)."""
    from xfastertransformer_b200.ops import native as Nat
    g = torch.Generator(device="cuda").manual_seed(T + I)
    x = torch.randn(T, K, generator=g, device="cuda").bfloat16()
    W = _linear(torch.randn(2 * I, K, generator=g, device="cuda") * 0.05, kind)
    gu = Nat.linear(x, W, out_dtype=None if kind == "w8a8" else torch.float32).double()
    want = torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]
    got = Nat.linear_gated(x, W, "silu").double()
    Nat.Workspace.get(x.device).check_status()
    assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -16 * gu.abs().amax()).all())


@pytest.mark.parametrize("T,I,K", [(1, 8, 64), (2, 72, 528), (16, 1096, 1040), (17, 200, 4096), (33, 136, 528), (64, 64, 2048), (100, 584, 272)])
def test_gated_uint4_ragged_features_match_64_bits(T, I, K):
    """Features that do not fill a tile of 64 gate and 64 up rows, one feature tile and many, with and without parts of k.  The products
    of either half are within the bound of `test_split_activations_match_64_bits`; |silu'| <= 1.1 and |silu(g)| <= |g| carry it on,
    and the result rounds to bf16."""
    from xfastertransformer_b200.ops import native as Nat
    g = torch.Generator(device="cuda").manual_seed(T + I + K)
    x = torch.randn(T, K, generator=g, device="cuda").bfloat16()
    W = _linear(torch.randn(2 * I, K, generator=g, device="cuda") * 0.05, "int4")
    w = R.dequant_weight(W).double()
    gu = x.double() @ w.t()
    tol = 2.0 ** -18 * (x.double().abs() @ (w.abs().t() + W.zero.double().abs()[None] * 2)) + \
        2.0 ** -21 * x.double().abs().amax(1, keepdim=True) * w.abs().sum(1)[None]
    want = torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]
    got = Nat.linear_gated(x, W, "silu").double()
    Nat.Workspace.get(x.device).check_status()
    bound = 1.1 * tol[:, :I] * gu[:, I:].abs() + (gu[:, :I].abs() + 1.1 * tol[:, :I]) * tol[:, I:] + 2.0 ** -8 * want.abs() + 2.0 ** -20
    assert bool(((got - want).abs() <= bound).all()), ((got - want).abs() / bound).max().item()


@pytest.mark.parametrize("T,N,K", [s for s in SHAPES if s[2] % 16 == 0] + [(300, 136, 144), (2300, 4104, 1024)])
def test_w8a8_sums_are_exact(T, N, K):
    """The integers that the tensor path sums, from the same codes: only the fp32 formula around the sum rounds."""
    from xfastertransformer_b200.ops import native as Nat
    from xfastertransformer_b200.ops import native_quant as Q
    g = torch.Generator(device="cuda").manual_seed(T * N)
    x = torch.randn(T, K, generator=g, device="cuda").bfloat16()
    W = _linear(torch.randn(N, K, generator=g, device="cuda") * 0.05, "w8a8")
    bias, res = torch.randn(N, generator=g, device="cuda"), torch.randn(T, N, generator=g, device="cuda").bfloat16()
    q, sa, za, qs = Q.quant_act(x, K)
    assert torch.equal(qs, q.float().sum(1))
    d = lambda t: t.double()
    terms = [d(sa)[:, None] * d(W.scale) * (d(q) @ d(W.w).t()), (d(sa) * d(qs))[:, None] * d(W.zero),
             d(za)[:, None] * (d(W.scale) * d(W.wsum)), K * d(za)[:, None] * d(W.zero), d(bias)[None], 0.5 * d(res)]
    got = Nat.linear(x, W, bias, None, res, 0.5, out_dtype=torch.float32)
    Nat.Workspace.get(x.device).check_status()
    assert bool(((d(got) - sum(terms)).abs() <= 2.0 ** -21 * sum(t.abs() for t in terms)).all())


@pytest.mark.parametrize("kind", ["int4", "fp8"])
def test_rows_that_are_not_finite_stay_alone(kind):
    from xfastertransformer_b200.ops import native as Nat
    x = torch.randn(20, 264, device="cuda").bfloat16()
    W = _linear(torch.randn(144, 264, device="cuda") * 0.05, kind)
    want = Nat.linear(x, W)
    y = x.clone()
    y[3, 5], y[7, 200], y[9, 263] = float("inf"), float("nan"), float("-inf")
    got = Nat.linear(y, W)
    bad = [3, 7, 9]
    keep = [i for i in range(20) if i not in bad]
    assert torch.equal(got[keep], want[keep]) and not torch.isfinite(got[bad]).any()


@pytest.mark.parametrize("T,E,k", [(1, 8, 2), (40, 8, 2), (90, 4, 2), (300, 4, 3)])
def test_fp8_experts_match_64_bits(T, E, k):
    from xfastertransformer_b200.ops import native as Nat
    g = torch.Generator(device="cuda").manual_seed(T)
    I, H = 256, 384
    experts = [(_linear(torch.randn(2 * I, H, generator=g, device="cuda") * 0.1, "fp8"), _linear(torch.randn(H, I, generator=g, device="cuda") * 0.1, "fp8"))
               for _ in range(E)]
    x = torch.randn(T, H, generator=g, device="cuda").bfloat16()
    idx = torch.rand(T, E - 1, generator=g, device="cuda").topk(k, 1)[1].int()              # one expert without tokens
    wt = torch.rand(T, k, generator=g, device="cuda") + 0.1
    want, tol = torch.zeros(T, H, dtype=torch.float64, device="cuda"), torch.zeros(T, H, dtype=torch.float64, device="cuda")
    for e, (a, b) in enumerate(experts):
        gu = x.double() @ R.dequant_weight(a).double().t()
        h = torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]
        d = R.dequant_weight(b).double()
        s = ((idx == e) * wt).sum(1, keepdim=True).double()
        want += s * (h @ d.t())
        tol += s * 2.0 ** -8 * (h.abs() @ d.abs().t())                                      # h is rounded to bf16
    got = Nat.moe_experts(x, idx, wt, experts).double()
    Nat.Workspace.get(x.device).check_status()
    assert bool(((got - want).abs() <= tol + 1e-5).all())


@pytest.mark.parametrize("kind", ["w8a8", "bf16"])
@pytest.mark.parametrize("T", [40, 66, 300])
@pytest.mark.parametrize("at", [1, 4])
def test_residual_that_starts_between_16_bytes(kind, T, at):
    """A slice of a wider tensor: its row pitch is a multiple of 16 bytes, its start is not.  The same bits as from a copy of it."""
    from xfastertransformer_b200.ops import native as Nat
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, 256, generator=g, device="cuda").bfloat16()
    W = _linear(torch.randn(512, 256, generator=g, device="cuda") * 0.05, kind)
    res = torch.randn(T, 520, generator=g, device="cuda").bfloat16()[:, at:at + 512]
    got, want = Nat.linear(x, W, None, None, res, 0.5), Nat.linear(x, W, None, None, res.contiguous(), 0.5)
    Nat.Workspace.get(x.device).check_status()
    assert torch.equal(got, want)


@pytest.mark.parametrize("nibbles", [False, True])
@pytest.mark.parametrize("top", [225.0, 288.0, 448.0, 450.0, 3.0e-20, 2.0e30])
def test_halves_of_an_activation(top, nibbles):
    """Every bf16 value up to a row's maximum: hi + lo / 16 times the row's scale is the value from 2^-13 of the maximum on, and at most
    2^-21 of it off below (the scaled maximum lies above 224, an e4m3 number ends at 2^-9, and lo is a sixteenth)."""
    from xfastertransformer_b200.ops import native_quant as Q
    v = torch.arange(0, 0x7F80, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    v = v[v.float() <= torch.tensor(top).bfloat16().float()]
    m = v.max().double()
    v = torch.cat([v, -v])[:(2 * v.numel()) // 32 * 32 if nibbles else None]
    v = torch.nn.functional.pad(v, (0, -v.numel() % 32)).view(1, -1)
    v[0, 0] = m.item()
    xs, scale, _ = Q.split_e4m3(v.cuda(), v.shape[1], nibbles)
    hi, lo = xs.cpu().view(torch.float8_e4m3fn).double().view(2, -1)
    got = (hi + lo / 16) * scale.cpu().double()
    if nibbles:                                                # 16 even ones, then 16 odd ones, of every 32
        got = got.view(-1, 2, 16).transpose(1, 2).reshape(-1)
    want = v[0].double()
    err = (got - want).abs()
    assert bool((err[want.abs() >= 2.0 ** -13 * m] == 0).all()) and bool((err <= 2.0 ** -21 * m).all())
