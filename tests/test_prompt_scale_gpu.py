"""Prompt attention with head_dim 128 and a softmax scale that is zero or negative, bf16 and int8 caches, plain and with a window: the largest score
is not that of the largest product then, and 0 x -inf is no score."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from xfastertransformer_b200.ops import reference as R


@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("scale", [0.0, -0.05, 0.05])
@pytest.mark.parametrize("window", [0, 100])
def test_any_sign(int8, scale, window):
    from xfastertransformer_b200.ops import native as N
    if int8 and window:
        pytest.skip("windows over an int8 cache have a kernel of their own")
    g = torch.Generator().manual_seed(7)
    lens, kv = [70, 130, 64], [70, 640, 65]
    blocks = [(n + 63) // 64 for n in kv]
    bt, at = torch.zeros(3, max(blocks), dtype=torch.int32), 1
    for i, n in enumerate(blocks):
        bt[i, :n] = torch.arange(at, at + n)
        at += n
    ks = vs = None
    if int8:
        kc, vc = (torch.randint(-127, 128, (at, 2, 64, 128), generator=g, dtype=torch.int8) for _ in range(2))
        ks, vs = (torch.rand(at, 2, 64, generator=g) * 0.02 + 1e-4 for _ in range(2))
        largest = float(vc.abs().amax() * vs.amax())
    else:
        kc, vc = (torch.randn(at, 2, 64, 128, generator=g).bfloat16() for _ in range(2))
        largest = float(vc.float().abs().amax())
    q = torch.randn(sum(lens), 8, 128, generator=g).bfloat16()
    cu = [0, 70, 200, 264]
    f = lambda t: t if t is None or t.dtype == torch.int8 else t.float()
    kw = dict(window=window) if window else {}
    want = R.paged_attention(q.float(), f(kc), f(vc), bt, cu, kv, scale, ks, vs, None, True, None, 4, 0, **kw)
    c = lambda t: None if t is None else t.cuda()
    got = N.paged_attention(c(q), c(kc), c(vc), c(bt), cu, kv, scale, c(ks), c(vs), None, True, None, 4, 0, **kw)
    N.Workspace.get(torch.device("cuda", 0)).check_status()
    # weights are rounded to bf16 (2^-9 each, they add up to one), the output too
    assert (got.float().cpu() - want).abs().max().item() <= 2.0 ** -7 * largest
