"""Decode steps whose keys are cut into slices: the CTAs of a cluster (up to eight) or apart (more), bf16 and int8 caches, slices without a
tile, query heads of several groups."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from xfastertransformer_b200.ops import reference as R


@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("splits", [1, 2, 3, 5, 8, 9])
@pytest.mark.parametrize("kv,hq,hkv", [([1, 64, 65, 600], 8, 2), ([129, 1500], 20, 1)])
def test_slices(int8, D, splits, kv, hq, hkv, monkeypatch):
    from xfastertransformer_b200.ops import native as N
    monkeypatch.setattr(N, "plan_attn_splits", lambda *a: (splits, 64))
    g = torch.Generator().manual_seed(sum(kv) + D)
    blocks = [(n + 63) // 64 for n in kv]
    nb = sum(blocks) + 1
    bt, at = torch.zeros(len(kv), max(blocks), dtype=torch.int32), 1
    for i, n in enumerate(blocks):
        bt[i, :n] = torch.arange(at, at + n)
        at += n
    ks = vs = None
    if int8:
        kc, vc = (torch.randint(-127, 128, (nb, hkv, 64, D), generator=g, dtype=torch.int8) for _ in range(2))
        ks, vs = (torch.rand(nb, hkv, 64, generator=g) * 0.02 + 1e-4 for _ in range(2))
        largest = float(vc.abs().amax() * vs.amax())
    else:
        kc, vc = (torch.randn(nb, hkv, 64, D, generator=g).bfloat16() for _ in range(2))
        largest = float(vc.float().abs().amax())
    q = torch.randn(len(kv), hq, D, generator=g).bfloat16()
    cu = list(range(len(kv) + 1))
    f = lambda t: t if t is None or t.dtype == torch.int8 else t.float()
    want = R.paged_attention(q.float(), f(kc), f(vc), bt, cu, kv, D ** -0.5, ks, vs, None, True, None, hq // hkv, 0)
    c = lambda t: None if t is None else t.cuda()
    got = N.paged_attention(c(q), c(kc), c(vc), c(bt), cu, kv, D ** -0.5, c(ks), c(vs), None, True, None, hq // hkv, 0)
    N.Workspace.get(torch.device("cuda", 0)).check_status()
    # weights are rounded to bf16 (2^-9 each, they add up to one), the output too
    assert (got.float().cpu() - want).abs().max().item() <= 2.0 ** -7 * largest
