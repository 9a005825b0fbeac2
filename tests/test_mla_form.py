"""Which prompts pay for the expanded form of latent attention: it works per visible key, the absorbed form per key and token."""
import pytest

from xfastertransformer_b200.ops.native_mla import expands


@pytest.mark.parametrize("new,past,want", [([64], [0], True), ([16] * 4, [0] * 4, True), ([16] * 4, [4000] * 4, False), ([16] * 4, [32000] * 4, False),
                                           ([32] * 8, [16000] * 8, False), ([64] * 4, [32000] * 4, True), ([2000], [0], True), ([128], [32000], True),
                                           ([63], [0], False), ([200, 3], [0, 9], False), ([300, 3], [0, 9], True), ([300, 3], [0, 90000], True)])
def test_by_tokens_and_visible_keys(new, past, want):
    cu = [0]
    for n in new:
        cu.append(cu[-1] + n)
    assert expands(cu, 128, 64, 512, 128, [a + b for a, b in zip(new, past)]) == want
