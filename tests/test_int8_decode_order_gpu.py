"""Decode steps over an int8 cache with heads of 128: the ring kernel gives the bits of the kernel that converts codes in shared memory (both in
csrc/kernels/attention.cu), whatever the number of slices, and so does either way of merging them."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from xfastertransformer_b200.utils.flags import Env


@pytest.mark.parametrize("splits", [None, 1, 2, 3, 5, 8, 9, 20])
@pytest.mark.parametrize("kv,hq,hkv", [([1, 31, 32, 33, 600], 8, 2), ([129, 1500], 20, 1), ([2870, 64, 17], 16, 16), ([17000], 8, 1)])
def test_ring_and_converting_kernel_agree(splits, kv, hq, hkv, monkeypatch):
    from xfastertransformer_b200.ops import native as N
    if splits is not None:
        monkeypatch.setattr(N, "plan_attn_splits", lambda *a: (splits, 32))
    g = torch.Generator(device="cuda").manual_seed(sum(kv) + hq)
    blocks = [(n + 63) // 64 for n in kv]
    nb = sum(blocks) + 1
    bt, at = torch.zeros(len(kv), max(blocks), dtype=torch.int32), 1
    for i, n in enumerate(blocks):
        bt[i, :n] = torch.arange(at, at + n)
        at += n
    kc, vc = (torch.randint(-127, 128, (nb, hkv, 64, 128), generator=g, device="cuda", dtype=torch.int8) for _ in range(2))
    ks, vs = (torch.rand(nb, hkv, 64, generator=g, device="cuda") * 0.02 + 1e-4 for _ in range(2))
    for b, n in enumerate(kv):                               # slots past the end hold whatever their last owner left
        for s in (ks, vs):
            s[bt[b, (n - 1) // 64], :, (n - 1) % 64 + 1:] = float("nan")
    q = torch.randn(len(kv), hq, 128, generator=g, device="cuda").bfloat16()
    bt = bt.cuda()

    def call():
        out = N.paged_attention(q, kc, vc, bt, list(range(len(kv) + 1)), kv, 128 ** -0.5, ks, vs, None, True, None, hq // hkv, 0)
        N.Workspace.get(q.device).check_status()
        return out

    ring = call()
    monkeypatch.setattr(Env.get(), "attn_tma", False)
    assert bool(ring.isfinite().all()) and torch.equal(ring, call())
