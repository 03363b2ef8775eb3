"""The tiles of the 32-bit product: every element is summed over k in order with one fused multiply-add a step, so each tile gives the bits
of the small one (which takes rows that do not start on 16 bytes)."""
import pytest
import torch

from miniserve_b200 import ops  # noqa: F401  (loads the kernels)
from miniserve_b200.ops import native

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _product(a, w, m, n, k, lda, ldw, batch=1):
    # (a width of whole fours and one more column: the last one belongs to nobody and stays as it is)
    out = torch.full((batch, m, n + 1), 7.0, device=DEV)
    code = native.kernels().ms_gemm_f32_batched(out.data_ptr(), a.data_ptr(), w.data_ptr(), m, n, k, lda, ldw, n + 1, batch,
                                                m * lda, n * ldw, m * (n + 1), torch.cuda.current_stream().cuda_stream)
    native.kernel_check(code)
    torch.cuda.synchronize()
    assert (out[..., n] == 7.0).all()
    return out[..., :n]


# tiles of 8 x 64, 32 x 32, 32 x 64, 80 x 64 and 64 x 128; the smallest, edges and one beside them, k that ends inside a step
@pytest.mark.parametrize("m, n, k, batch", [
    (1, 1, 65, 1), (8, 19000, 100, 1), (9, 9501, 68, 1), (1, 700, 96, 16),
    (33, 1025, 72, 1), (96, 1057, 127, 1), (31, 33, 130, 9),
    (64, 8192, 96, 1), (65, 4095, 97, 1),
    (80, 9472, 100, 1), (700, 1024, 132, 1), (721, 1027, 95, 1),
    (700, 4096, 80, 1), (129, 20000, 81, 1), (513, 511, 66, 8),
])
def test_every_tile_gives_the_same_bits(m, n, k, batch):
    torch.manual_seed(m + n)
    lda = (k + 3) // 4 * 4
    a = torch.full((batch, m, lda), float("nan"), device=DEV)  # (what lies behind the last k is not read into a sum)
    w = torch.full((batch, n, lda), float("nan"), device=DEV)
    a[..., :k], w[..., :k] = torch.randn(batch, m, k, device=DEV), torch.randn(batch, n, k, device=DEV)
    out = _product(a, w, m, n, k, lda, lda, batch)
    odd_a, odd_w = (torch.zeros(batch, x.shape[1], lda + 1, device=DEV) for x in (a, w))
    odd_a[..., :k], odd_w[..., :k] = a[..., :k], w[..., :k]
    small = _product(odd_a, odd_w, m, n, k, lda + 1, lda + 1, batch)
    assert torch.equal(out, small)
    exact = a[..., :k].double() @ w[..., :k].double().transpose(1, 2)
    # (k roundings of partial sums, each below 2^-24 of the sum of the products' sizes)
    size = a[..., :k].double().abs() @ w[..., :k].double().abs().transpose(1, 2)
    assert ((out.double() - exact).abs() <= k * 2.0 ** -24 * size).all()
