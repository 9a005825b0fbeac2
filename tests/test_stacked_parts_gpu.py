"""Gated uint4 products whose tiles stack both halves (csrc/kernels/gemm_e4m3_sm100.cu): k is cut into the parts that 64 rows have, so a row's bits do
not depend on the rows beside it."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from xfastertransformer_b200.runtime.loader import make_linear


def _weights(rows, K, kind, g):
    return make_linear(torch.randn(rows, K, generator=g, device="cuda") * 0.05, kind).to("cuda")


@pytest.mark.parametrize("T", [1, 16, 32])
@pytest.mark.parametrize("I", [1928, 2048, 2112, 4352, 4480, 4544])
def test_stacked_uint4_tiles_are_cut_as_64_rows_are(T, I):
    """Feature counts around the lines at which a product is cut into more parts of k."""
    from xfastertransformer_b200.ops import native as N
    g = torch.Generator(device="cuda").manual_seed(T + I)
    x = torch.randn(64, 4096, generator=g, device="cuda").bfloat16()
    W = _weights(2 * I, 4096, "int4", g)
    assert torch.equal(N.linear_gated(x[:T].contiguous(), W), N.linear_gated(x, W)[:T])
