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


# the packer's tables begin with the page ahead of the window's first (given back: -1); a tile of 32 keys may begin several pages ahead of that
@pytest.mark.parametrize("page", [1, 4, 8, 16, 32])
@pytest.mark.parametrize("window, keep_first", [(1, 0), (5, 0), (7, 9), (40, 0)])
def test_tables_that_begin_behind_a_tile(page, window, keep_first):
    torch.manual_seed(page + window)
    rows, nq, nkv, d = [(70, 33), (0, 45), (131, 9), (95, 64)], 5, 1, 32
    pb = PagedBatch(rows, page, nkv, d, torch.float32, seed=3)
    for r, (s, n) in enumerate(rows):
        pb.fill(r, torch.randn(s + n, nkv, d, device=DEV), torch.randn(s + n, nkv, d, device=DEV))
    ctx, q = make_context(pb), torch.randn(pb.num_tokens, nq, d, device=DEV)
    extras = ops.AttentionExtras(None, 0.0, 0, None, None, keep_first)
    want, got = (torch.full_like(q, float("nan")) for _ in range(2))
    ops.attention_rowwise(want, q, pb.k_pool, pb.v_pool, ctx.positions, ctx.row_of_token, ctx.page_indptr[0], ctx.page_indices[0], 0.3, window, ctx.status,
                          extras=extras)
    indices, indptr, nowhere = [], [], [1 << 28] * 40  # (what lies ahead of a row's table is no page)
    for (s, _), table in zip(rows, pb.tables):
        live = 0 if keep_first else max(0, s - window + 1) // page
        begin = max(live - 1, 0)
        indices += nowhere
        indptr.append(len(indices) - begin)
        indices += ([-1] if live else []) + table[live:]
    ctx.page_indptr[0] = torch.tensor(indptr + [len(indices)], dtype=torch.int32, device=DEV)
    ctx.page_indices[0] = torch.tensor(indices, dtype=torch.int32, device=DEV)
    assert ops.attention_tiled_ok(got, q, pb.k_pool, pb.v_pool, ctx)
    ops.attention_tiled(got, q, pb.k_pool, pb.v_pool, ctx, 0, 0.3, window, extras=extras)
    assert ctx.status.item() == 0 and torch.equal(got, want)
