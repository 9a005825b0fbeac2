"""Prompt attention with head_dim 128 on the tensor cores (csrc/kernels/attention_prefill_sm100.cu) over a bf16 cache, against the plain
formulation: rows and keys that end inside and at the edges of its tiles of 128 and chunks of 16 and 32."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from xfastertransformer_b200.ops import reference as R


@pytest.mark.parametrize("lens,past", [([16, 17, 31, 32, 33], [0] * 5), ([63, 64, 65, 127], [0, 1, 63, 64]), ([128, 129, 256, 257], [0] * 4),
                                       ([2, 1, 130], [500, 0, 127]), ([700], [0]), ([20, 300], [1000, 333])])
@pytest.mark.parametrize("hq,hkv", [(4, 4), (8, 2)])
def test_prompts(lens, past, hq, hkv):
    from xfastertransformer_b200.ops import native as N
    g = torch.Generator().manual_seed(sum(lens) + hq)
    kv = [n + p for n, p in zip(lens, past)]
    blocks = [(n + 63) // 64 for n in kv]
    nb = sum(blocks) + 3
    perm = (torch.randperm(nb - 1, generator=g) + 1).tolist()
    bt, at = torch.zeros(len(lens), max(blocks) + 2, dtype=torch.int32), 0
    for i, n in enumerate(blocks):
        bt[i, :n] = torch.tensor(perm[at:at + n], dtype=torch.int32)
        at += n
    kc, vc = (torch.randn(nb, hkv, 64, 128, generator=g).bfloat16() for _ in range(2))
    q = (torch.randn(sum(lens), hq, 128, generator=g) * 2).bfloat16()
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    want = R.paged_attention(q.float(), kc.float(), vc.float(), bt, cu, kv, 128 ** -0.5, None, None, None, True, None, hq // hkv, 0)
    got = N.paged_attention(q.cuda(), kc.cuda(), vc.cuda(), bt.cuda(), cu, kv, 128 ** -0.5, None, None, None, True, None, hq // hkv, 0)
    N.Workspace.get(torch.device("cuda", 0)).check_status()
    # a weight is rounded to bf16 (2^-9 of it; they add up to one), the output too
    tol = 2.0 ** -8 * float(vc.float().abs().amax())
    err = (got.float().cpu() - want).abs().max().item()
    assert err <= tol, (err, tol)
