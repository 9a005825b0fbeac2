"""Attention over an int8 cache: prompts on the tensor cores through a copy of the codes (head_dim 128), and decode steps whose tiles
are fetched ahead, against the plain formulation."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from xfastertransformer_b200.ops import reference as R


def _run(lens, past, hq, hkv, D, seed, monkeypatch, never=False, stale=None):
    from xfastertransformer_b200.ops import native as N
    monkeypatch.setattr(N, "INT8_TC_MIN_KV", 1 << 30 if never else 0)
    g = torch.Generator().manual_seed(seed)
    kv = [n + p for n, p in zip(lens, past)]
    blocks = [(n + 63) // 64 for n in kv]
    nb = sum(blocks) + 3
    perm = (torch.randperm(nb - 1, generator=g) + 1).tolist()
    bt, at = torch.zeros(len(lens), max(blocks) + 2, dtype=torch.int32), 0
    for i, n in enumerate(blocks):
        bt[i, :n] = torch.tensor(perm[at:at + n], dtype=torch.int32)
        at += n
    kc, vc = (torch.randint(-127, 128, (nb, hkv, 64, D), generator=g, dtype=torch.int8) for _ in range(2))
    ks, vs = (torch.rand(nb, hkv, 64, generator=g) * 0.02 + 1e-4 for _ in range(2))
    largest = float((vc.abs().amax() * vs.amax()))
    if stale is not None:                                    # scales of slots that hold no key of these sequences
        for i, n in enumerate(kv):
            if n % 64:
                for t in (ks, vs):
                    t[int(bt[i, blocks[i] - 1]), :, n % 64:] = stale
    q = torch.randn(sum(lens), hq, D, generator=g).bfloat16()
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    scale = D ** -0.5
    want = R.paged_attention(q.float(), kc, vc, bt, cu, kv, scale, ks, vs, None, True, None, hq // hkv, 0)
    c = lambda t: t.cuda()
    got = N.paged_attention(c(q), c(kc), c(vc), c(bt), cu, kv, scale, c(ks), c(vs), None, True, None, hq // hkv, 0)
    N.Workspace.get(torch.device("cuda", 0)).check_status()
    # weights are rounded to bf16 (2^-9 each, they add up to one), the output too
    tol = 2.0 ** -7 * largest
    err = (got.float().cpu() - want).abs().max().item()
    assert err <= tol, (err, tol)


# one past the copy's threshold, tiles of 128 rows and keys cut at their edges, prompts behind cached tokens, one short one among long
@pytest.mark.parametrize("lens,past", [([64], [0]), ([128, 129, 65], [0, 0, 0]), ([200, 1, 77], [0, 64, 300]), ([300], [127]),
                                       ([65, 256], [1, 512])])
@pytest.mark.parametrize("hq,hkv", [(4, 4), (8, 2)])
def test_prompts(lens, past, hq, hkv, monkeypatch):
    _run(lens, past, hq, hkv, 128, sum(lens), monkeypatch)


def test_prompt_without_the_copy(monkeypatch):
    _run([130, 70], [0, 40], 8, 2, 128, 5, monkeypatch, never=True)


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("kv", [[1], [16, 17, 31], [33, 64, 65, 127], [300, 900, 2049]])
def test_steps(D, kv, monkeypatch):
    _run([1] * len(kv), [n - 1 for n in kv], 8, 2, D, D + sum(kv), monkeypatch)


@pytest.mark.parametrize("stale", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("lens,past", [([65], [0]), ([100, 190, 64], [0, 3, 1]), ([1, 1], [99, 700])])
def test_scales_past_the_end(stale, lens, past, monkeypatch):
    """Slots of the last block beyond a sequence's length keep what an earlier owner left there, overflowed values too."""
    _run(lens, past, 8, 2, 128, sum(lens), monkeypatch, stale=stale)


def test_prompt_on_a_full_card(monkeypatch):
    """Where the copy of the codes has no room, the kernel that reads them where they are takes the prompt, as it did all of them."""
    empty, refused = torch.empty, []

    def short(*size, **kw):
        if len(size) == 5 and kw.get("dtype") == torch.bfloat16:
            refused.append(size)
            raise torch.OutOfMemoryError("no room")
        return empty(*size, **kw)
    monkeypatch.setattr(torch, "empty", short)
    _run([130, 70], [0, 40], 8, 2, 128, 5, monkeypatch)
    assert refused
