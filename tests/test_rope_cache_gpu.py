"""Split + rotation + cache append: the kernel of whole heads in pairs (i, i + D/2) against the general one, bit for bit."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _both(T, hq, hkv, D, int8, scale, seed):
    """(fast, general): the general kernel is reached through a row pitch that 16-byte loads do not fit."""
    from xfastertransformer_b200.ops import native as N
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = (hq + 2 * hkv) * D
    base = torch.randn(T, n + 12, generator=g, device="cuda").bfloat16()
    base[0, :n] = 0
    pos = torch.randint(0, 500, (T,), generator=g, device="cuda").int()
    table = torch.randn(500, D, generator=g, device="cuda")
    nb = (T + 63) // 64 + 2
    slots = torch.randperm(nb * 64, generator=g, device="cuda")[:T].int()
    qs = torch.rand(T, generator=g, device="cuda") + 0.5 if scale else None
    outs = []
    for ld, rows in ((n, base[:, :n].contiguous()), (n + 12, base)):
        dt = torch.int8 if int8 else torch.bfloat16
        kc, vc = (torch.zeros(nb, max(hkv, 1), 64, D, dtype=dt, device="cuda") for _ in range(2))
        ks, vs = (torch.zeros(nb, max(hkv, 1), 64, device="cuda") for _ in range(2))
        q = torch.empty(T, hq, D, dtype=torch.bfloat16, device="cuda")
        ws = N.Workspace.get(q.device)
        rc = N.lib().xft_qkv_rope_cache(N._p(rows), ld, T, hq, hkv, D, N._p(pos), N._p(table), D, 0, 0, 500, N._p(qs), N._p(None), N._p(None),
                                        C.c_float(1e-6), N._p(q), N._p(kc), N._p(vc), N._p(ks if int8 else None), N._p(vs if int8 else None),
                                        int(int8), 64, C.c_longlong(nb * 64), N._p(slots), N._p(ws.status), N._stream())
        assert rc == 0
        ws.check_status()
        outs.append((q, kc, vc, ks, vs))
    return outs


# one token; heads that do not fill a warp or a group of four; enough for four heads per thread
@pytest.mark.parametrize("T,hq,hkv", [(1, 4, 4), (3, 5, 1), (67, 9, 2), (2100, 32, 8), (5, 3, 0)])
@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("int8,scale", [(False, False), (True, False), (False, True)])
def test_same_bits_as_the_general_kernel(T, hq, hkv, D, int8, scale):
    fast, general = _both(T, hq, hkv, D, int8, scale, T + D)
    for a, b in zip(fast, general):
        assert torch.equal(a, b)
