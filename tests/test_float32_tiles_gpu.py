"""The large-tile forms of the 32-bit kernels give the bits of the small ones: matrix products against the same rows a few at a time,
prompt attention against the row-wise kernel, with every extra, over odd sizes, ragged rows, portions and pages that were given back."""

import pytest
import torch

from miniserve_b200 import ops
from tests.kernel_util import PagedBatch, make_context

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")


@pytest.mark.parametrize("m, n, k", [(33, 1, 1), (64, 128, 16), (65, 129, 17), (700, 1024, 130), (700, 4096, 64), (1500, 1000, 35), (2048, 2048, 48), (257, 96, 1000)])
@pytest.mark.parametrize("pad", [0, 1])
def test_products_in_large_tiles_are_the_small_ones_bit_for_bit(m, n, k, pad):
    gen = torch.Generator(device=DEV).manual_seed(m + n + k)
    # (pad: rows that do not start on 16 bytes)
    x, w = (torch.randn(r * k + pad, generator=gen, device=DEV)[pad:].view(r, k) for r in (m, n))
    got = torch.full((m, n), float("nan"), device=DEV)
    ops.linear(x, w, out=got)
    small = torch.cat([ops.linear(x[a:a + 32].contiguous(), w) for a in range(0, m, 32)])  # up to 32 rows: the small tiles
    assert torch.equal(got, small)
    assert (got.double() - x.double() @ w.double().T).abs().max() < 1e-5 * k ** 0.5 * 5


@pytest.mark.parametrize("heads, k, n", [(3, 64, 96), (2, 33, 130)])
def test_products_of_heads_in_large_tiles(heads, k, n):
    t = 200
    x = torch.randn(t, heads, k, device=DEV)
    w = torch.randn(heads, n, k, device=DEV)
    got = torch.empty(t, heads, n, device=DEV)
    ops.linear_heads(x, w, got)
    for h in range(heads):
        assert torch.equal(got[:, h], ops.linear(x[:, h].contiguous(), w[h].contiguous()))


EXTRAS = {"plain": {}, "window": dict(window=50), "sink": dict(sink=True), "learned": dict(learned=True), "softcap": dict(softcap=8.0),
          "chunk": dict(chunk=48, window=48), "distance": dict(distance=True), "kept": dict(window=40, keep_first=5, distance=True, learned=True)}


@pytest.mark.parametrize("extra", sorted(EXTRAS))
@pytest.mark.parametrize("nq, nkv, d, page", [(4, 2, 128, 16), (6, 1, 20, 4), (3, 3, 64, 8), (10, 2, 100, 32)])
def test_prompt_attention_in_tiles_is_the_row_wise_one_bit_for_bit(extra, nq, nkv, d, page):
    e = EXTRAS[extra]
    rows = [(0, 1), (0, 130), (77, 65), (300, 3), (0, 32), (31, 1), (5, 64)]
    torch.manual_seed(nq * d)
    pb = PagedBatch(rows, page, nkv, d, torch.float32, seed=3)
    for r, (s, n) in enumerate(rows):
        pb.fill(r, torch.randn(s + n, nkv, d, device=DEV), torch.randn(s + n, nkv, d, device=DEV))
    ctx = make_context(pb)
    window, chunk = e.get("window"), e.get("chunk", 0)
    if window and not e.get("keep_first") and not chunk:
        # pages behind every window may have been given back: the table says so, nothing may look there
        table = pb.page_indices.tolist()
        at = 0
        for (s, n), t in zip(rows, pb.tables):
            for p in range(max(0, (s - window + 1)) // page):
                table[at + p] = -1
            at += len(t)
        ctx.page_indices[0] = torch.tensor(table, dtype=torch.int32, device=DEV)
    q = torch.randn(pb.num_tokens, nq, d, device=DEV) * 2
    extras = ops.AttentionExtras(torch.randn(nq, device=DEV) if e.get("learned") else None, e.get("softcap", 0.0), chunk,
                                 torch.rand(nq, device=DEV) if e.get("distance") else None, torch.rand(nq, device=DEV) + 0.1 if e.get("distance") else None,
                                 e.get("keep_first", 0))
    want, got = (torch.full_like(q, float("nan")) for _ in range(2))
    ops.attention_rowwise(want, q, pb.k_pool, pb.v_pool, ctx.positions, ctx.row_of_token, ctx.page_indptr[0], ctx.page_indices[0], d ** -0.5, window,
                          ctx.status, sink=e.get("sink", False), extras=extras)
    assert ops.attention_tiled_ok(got, q, pb.k_pool, pb.v_pool, ctx)
    ops.attention(got, q, pb.k_pool, pb.v_pool, ctx, 0, d ** -0.5, window, e.get("sink", False), extras)
    assert ctx.status.item() == 0 and not torch.isnan(want).any() and torch.equal(got, want)


def test_a_page_that_is_missing_raises_the_status_word():
    pb = PagedBatch([(0, 40)], 8, 1, 32, torch.float32)
    pb.fill(0, torch.randn(40, 1, 32, device=DEV), torch.randn(40, 1, 32, device=DEV))
    ctx = make_context(pb)
    ctx.page_indices[0][2] = -1
    q = torch.randn(40, 2, 32, device=DEV)
    ops.attention(torch.empty_like(q), q, pb.k_pool, pb.v_pool, ctx, 0, 0.2, None)
    assert ctx.status.item() == 3
