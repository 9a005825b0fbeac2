"""Row sums in front of products of int8 weights (csrc/kernels/quant_gemm_sm100.cu): added in strides of 256, then by lanes, then by warps."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [8, 200, 256, 1000, 4096, 11008])
def test_row_sums_go_in_strides_of_256(K):
    from xfastertransformer_b200.ops import native_quant as Q
    x = torch.randn(5, K, generator=torch.Generator(device="cuda").manual_seed(K), device="cuda").bfloat16()
    f = torch.nn.functional.pad(x.float(), (0, -K % 256)).view(5, -1, 256)
    v = torch.zeros(5, 256, device="cuda")
    for i in range(f.shape[1]):
        v = v + f[:, i]
    v = v.view(5, 8, 32)
    lane = torch.arange(32, device="cuda")
    for o in (16, 8, 4, 2, 1):
        v = v + v[..., lane ^ o]
    want = torch.zeros(5, device="cuda")
    for w in range(8):
        want = want + v[:, w, 0]
    assert torch.equal(Q._row_sums(x, K), want)
