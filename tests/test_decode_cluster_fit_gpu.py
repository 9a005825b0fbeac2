"""Decode steps whose slices would need more clusters than the GPU takes at a time are merged through scratch: the bits of few sequences, whose
slices share clusters."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("splits", [2, 4, 5, 8])
def test_many_sequences_and_few(int8, D, splits, monkeypatch):
    from xfastertransformer_b200.ops import native as N
    monkeypatch.setattr(N, "plan_attn_splits", lambda *a: (splits, 64))
    g = torch.Generator(device="cuda").manual_seed(D + splits)
    B, hkv, hq = 150, 2, 8
    kv = [1 + 29 * i % 1200 for i in range(B)]
    bt = (torch.arange(B * 19, dtype=torch.int32, device="cuda") % 200).view(B, 19)      # pages may be shared: they are only read
    ks = vs = None
    if int8:
        kc, vc = (torch.randint(-127, 128, (200, hkv, 64, D), generator=g, device="cuda", dtype=torch.int8) for _ in range(2))
        ks, vs = (torch.rand(200, hkv, 64, generator=g, device="cuda") * 0.02 + 1e-4 for _ in range(2))
    else:
        kc, vc = (torch.randn(200, hkv, 64, D, generator=g, device="cuda").bfloat16() for _ in range(2))
    q = torch.randn(B, hq, D, generator=g, device="cuda").bfloat16()

    def call(i, j):
        return N.paged_attention(q[i:j], kc, vc, bt[i:j], list(range(j - i + 1)), kv[i:j], D ** -0.5, ks, vs, None, True, None, hq // hkv, 0)

    whole = call(0, B)
    for i in range(0, B, 6):
        assert torch.equal(whole[i:i + 6], call(i, i + 6))
    N.Workspace.get(q.device).check_status()
