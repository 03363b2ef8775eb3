"""The packer's page tables begin with the page ahead of a window's first one; tensor-core attention walks tiles of 64 and 128 keys, which may begin further
back. What stands ahead of a row's table changes nothing."""
import pytest
import torch

from miniserve_b200 import ops
from tests.kernel_util import PagedBatch, make_context

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")


@pytest.mark.parametrize("page", [8, 16, 32])
@pytest.mark.parametrize("window, keep_first", [(5, 0), (40, 0), (200, 0), (33, 9)])
@pytest.mark.parametrize("d", [64, 128])
def test_numbers_ahead_of_a_table(page, window, keep_first, d):
    torch.manual_seed(page + window)
    rows, nq, nkv = [(700, 133), (0, 245), (431, 19), (255, 64), (900, 1)], 4, 2
    pb = PagedBatch(rows, page, nkv, d, torch.bfloat16, seed=3)
    for r, (s, n) in enumerate(rows):
        pb.fill(r, torch.randn(s + n, nkv, d, device=DEV).bfloat16(), torch.randn(s + n, nkv, d, device=DEV).bfloat16())
    ctx, q = make_context(pb), torch.randn(pb.num_tokens, nq, d, device=DEV).bfloat16()
    extras = ops.AttentionExtras(None, 0.0, 0, None, None, keep_first) if keep_first else None
    want, got = (torch.full_like(q, float("nan")) for _ in range(2))
    ops.attention(want, q, pb.k_pool, pb.v_pool, ctx, 0, 0.1, window, extras=extras)
    indices, indptr = [], []
    for (s, _), table in zip(rows, pb.tables):
        live = 0 if keep_first else max(0, s - window + 1) // page
        indices += [1 << 28] * 40
        indptr.append(len(indices) - max(live - 1, 0))
        indices += ([-1] if live else []) + table[live:]
    ctx.page_indptr[0] = torch.tensor(indptr + [len(indices)], dtype=torch.int32, device=DEV)
    ctx.page_indices[0] = torch.tensor(indices, dtype=torch.int32, device=DEV)
    ops.attention(got, q, pb.k_pool, pb.v_pool, ctx, 0, 0.1, window, extras=extras)
    assert ctx.status.item() == 0 and torch.isfinite(got).all() and torch.equal(got, want)
