"""Slices of a decode step (ops/native.py): long contexts over an int8 cache are cut as finely as the CTA slots allow, and the plan is one for all
kernels of such a cache."""
import pytest

from xfastertransformer_b200.ops import native as N


@pytest.mark.parametrize("B,hkv,group,max_kv,want", [(1, 8, 4, 600, 2), (1, 8, 4, 8000, 31), (1, 8, 4, 32000, 32), (2, 8, 4, 32000, 18), (4, 1, 8, 32000, 32),
                                                     (40, 1, 40, 3000, 2), (8, 8, 4, 2870, 4), (8, 5, 8, 3000, 7), (64, 8, 8, 200, 1)])
def test_int8_slices(B, hkv, group, max_kv, want):
    """296 slots, at least eight tiles of 32 keys each, 32 slices at most."""
    assert N.plan_attn_splits(B, hkv, group, 128, max_kv, True) == (want, (max_kv + 31) // 32)
