"""Form of DeepSeek's latent attention in prompts (ops/native_mla.py): absorbed unless XFT_MLA_EXPAND asks for the other, whatever layout the queries
come in."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from test_mla_prompt_gpu import _check, _inputs
from xfastertransformer_b200.utils.flags import Env


@pytest.mark.parametrize("lens,past", [([64], [0]), ([97, 128, 70], [0, 0, 500]), ([16, 16, 16, 16], [900, 0, 64, 1])])
@pytest.mark.parametrize("packed", [True, False])
def test_prompts_are_absorbed(lens, past, packed):
    from xfastertransformer_b200.ops import native as Nat
    from xfastertransformer_b200.ops import native_mla
    cache, bt, cu, kv, q, wk, wv = (t.cuda() if isinstance(t, torch.Tensor) else t for t in _inputs(lens, past, 16))
    qn, qr = q[..., :128], q[..., 128:]
    if not packed:
        qn, qr = qn.transpose(0, 1).contiguous().transpose(0, 1), qr.contiguous()
    dev = q.device
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)
    got = Nat.mla_attention(qn, qr, cache, bt, cu, kv, wk, wv, 192 ** -0.5)
    want = native_mla._absorbed(qn, qr, cache, bt, i32(cu), i32(kv), len(kv), max(kv), wk, wv, 192 ** -0.5, None)
    Nat.Workspace.get(dev).check_status()
    assert torch.equal(got, want)


@pytest.mark.parametrize("lens,past", [([64], [0]), ([127, 128, 129], [0, 0, 0]), ([255, 257, 16], [0, 1, 64]), ([200, 3, 1, 90], [0, 50, 9, 77])])
@pytest.mark.parametrize("packed", [True, False])
def test_expanded_where_asked_for(lens, past, packed, monkeypatch):
    from xfastertransformer_b200.ops import native_mla
    monkeypatch.setattr(Env.get(), "mla_expand", True)
    calls = []
    expanded = native_mla._expanded
    monkeypatch.setattr(native_mla, "_expanded", lambda *a: calls.append(1) or expanded(*a))
    _check(lens, past, 16, packed)
    assert calls
