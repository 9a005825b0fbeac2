"""Latent attention of prompts in the expanded form (ops/native_mla.py): portions at the edges of its tiles, behind cached tokens, beside
portions too short for it, queries in both layouts, heads in turns and without room for the expanded keys."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

from xfastertransformer_b200.ops import reference as R


def _inputs(lens, past, Hl, seed=3):
    g = torch.Generator().manual_seed(seed + sum(lens) + Hl)
    kv = [a + b for a, b in zip(lens, past)]
    nbs = [(n + 63) // 64 for n in kv]
    nb = sum(nbs) + 1
    perm = torch.randperm(nb, generator=g).tolist()
    bt, at = torch.zeros(len(lens), max(nbs), dtype=torch.int32), 0
    for b, n in enumerate(nbs):
        bt[b, :n] = torch.tensor(perm[at:at + n], dtype=torch.int32)
        at += n
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    r = lambda *s, f=0.5: (torch.randn(*s, generator=g) * f).bfloat16()
    return r(nb, 1, 64, 576), bt, cu, kv, r(cu[-1], Hl, 192), r(Hl, 128, 512, f=0.06), r(Hl, 128, 512, f=0.06)


def _check(lens, past, Hl, packed=True):
    from xfastertransformer_b200.ops import native as Nat
    from xfastertransformer_b200.ops import native_mla
    cache, bt, cu, kv, q, wk, wv = _inputs(lens, past, Hl)
    assert native_mla.expands(cu, 128, 64, 512, 128)
    scale = 1 / math.sqrt(192)
    want = R.mla_attention(q[..., :128].float(), q[..., 128:].float(), cache, bt, cu, kv, wk, wv, scale, absorbed=False)
    qc = q.cuda()
    qn, qr = qc[..., :128], qc[..., 128:]
    if not packed:
        qn, qr = qn.transpose(0, 1).contiguous().transpose(0, 1), qr.contiguous()
    got = Nat.mla_attention(qn, qr, cache.cuda(), bt.cuda(), cu, kv, wk.cuda(), wv.cuda(), scale)
    Nat.Workspace.get(torch.device("cuda", 0)).check_status()
    # keys, values, weights and output are rounded to bf16 (2^-9 each); a rounded key moves a weight by its score's change,
    # 2^-9 |q| |k| / sqrt(192) at most and about 2^-9 of the largest score of some 5 in all
    assert (got.float().cpu() - want).abs().max().item() <= 2.0 ** -6 * want.abs().max().item()


@pytest.mark.parametrize("lens,past", [([64], [0]), ([127, 128, 129], [0, 0, 0]), ([255, 257, 16], [0, 1, 64]), ([70, 64], [1000, 63])])
@pytest.mark.parametrize("Hl", [8, 40])
@pytest.mark.parametrize("packed", [True, False])
def test_portions(lens, past, Hl, packed):
    _check(lens, past, Hl, packed)


def test_beside_short_portions():
    _check([200, 3, 1, 90], [0, 50, 9, 77], 16)


def test_heads_in_turns(monkeypatch):
    from xfastertransformer_b200.ops import native_latent
    monkeypatch.setattr(native_latent, "EXPAND_BYTES", 2 * 300 * 256 * 3)        # three heads at a time
    _check([300], [0], 8)


def test_without_room(monkeypatch):
    """Where the expanded keys and values have no room the absorbed form takes the prompt, as it did all of them."""
    from xfastertransformer_b200.ops import native_mla
    monkeypatch.setattr(native_mla, "_expanded", lambda *a: False)
    _check([100, 64], [0, 7], 8)
