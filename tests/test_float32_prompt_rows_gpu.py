"""32-bit prompt attention in its two heights of tile (32 and 64 query rows), and over grids of more than two tiles a multiprocessor: the
bits of the row-wise kernel."""
import pytest
import torch

from miniserve_b200 import ops
from tests.kernel_util import PagedBatch, make_context

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")


# groups of 1 to 32 heads take 32 rows where that leaves no more of them idle, the others 64; steps are pairs of 32 keys: an odd last tile,
# a first tile behind a window, kept keys whose tiles end one pair early
@pytest.mark.parametrize("nq, nkv, d", [(32, 1, 128), (20, 1, 32), (64, 1, 128), (48, 1, 68), (8, 8, 36)])
@pytest.mark.parametrize("window, keep_first, softcap", [(None, 0, 0.0), (70, 0, 9.0), (45, 33, 0.0)])
def test_both_heights(nq, nkv, d, window, keep_first, softcap):
    _compare([(0, 33), (0, 97), (130, 31), (64, 64), (0, 2), (200, 1)], nq, nkv, d, window, ops.AttentionExtras(None, softcap, 0, None, None, keep_first))


# tiles of 16 tokens (8 kv heads, 2 heads each): 37 of them fill 296 places with the second half turned round; one fewer does not
@pytest.mark.parametrize("rows", [[(0, 592)], [(0, 575)], [(0, 900)], [(0, 300), (20, 290), (0, 17)]])
def test_the_order_of_the_grid(rows):
    _compare(rows, 16, 8, 128, None, ops.AttentionExtras(None, 0.0, 0, None, None, 0))


def _compare(rows, nq, nkv, d, window, extras):
    torch.manual_seed(nq * d)
    pb = PagedBatch(rows, 16, nkv, d, torch.float32, seed=3)
    for r, (s, n) in enumerate(rows):
        pb.fill(r, torch.randn(s + n, nkv, d, device=DEV), torch.randn(s + n, nkv, d, device=DEV))
    ctx = make_context(pb)
    q = torch.randn(pb.num_tokens, nq, d, device=DEV) * 2
    want, got = (torch.full_like(q, float("nan")) for _ in range(2))
    ops.attention_rowwise(want, q, pb.k_pool, pb.v_pool, ctx.positions, ctx.row_of_token, ctx.page_indptr[0], ctx.page_indices[0], d ** -0.5, window,
                          ctx.status, extras=extras)
    assert ops.attention_tiled_ok(got, q, pb.k_pool, pb.v_pool, ctx)
    ops.attention_tiled(got, q, pb.k_pool, pb.v_pool, ctx, 0, d ** -0.5, window, extras=extras)
    assert ctx.status.item() == 0 and torch.equal(got, want)
