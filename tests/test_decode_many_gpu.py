"""Decode steps with more (sequence, kv head) pairs than resident CTAs: the walking kernel against the kernel with a CTA per pair (the
same batch in pieces small enough for it), bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,hkv,group,longest", [(75, 4, 1, 300), (10, 32, 1, 1100), (40, 8, 4, 200), (300, 1, 2, 70), (500, 2, 3, 129)])
def test_same_bits_as_a_cta_per_pair(B, hkv, group, longest, D, monkeypatch):
    from xfastertransformer_b200.models.decoder import Batch
    from xfastertransformer_b200.ops import native as N
    monkeypatch.setattr(N, "BRIEF_KV", 1 << 30)
    g = torch.Generator().manual_seed(B + D)
    kv = torch.randint(1, longest + 1, (B,), generator=g).tolist()
    kv[:4] = [1, 64, 65, longest]
    W = (longest + 63) // 64
    nb = B * W
    bt = torch.randperm(nb, generator=g).int().view(B, W).cuda()
    kc, vc = (torch.randn(nb, hkv, 64, D, generator=g).bfloat16().cuda() for _ in range(2))
    q = torch.randn(B, hkv * group, D, generator=g).bfloat16().cuda()
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")

    def run(a, e):
        n = e - a
        b = Batch(ids=None, positions=None, slots=None, cu_q=list(range(n + 1)), kv_lens=kv[a:e], block_table=bt[a:e], is_decode=True, max_q=1,
                  max_kv=max(kv[a:e]))
        b.cu_q_dev, b.kv_lens_dev = i32(list(range(n + 1))), i32(kv[a:e])
        b.meta["nsplit"] = 1
        return N.paged_attention(q[a:e], kc, vc, bt[a:e], b.cu_q, b.kv_lens, D ** -0.5, group=group, meta=b)

    assert B * hkv > 296
    got = run(0, B)
    step = 296 // hkv
    want = torch.cat([run(a, min(a + step, B)) for a in range(0, B, step)])
    N.Workspace.get(q.device).check_status()
    assert torch.equal(got, want)
