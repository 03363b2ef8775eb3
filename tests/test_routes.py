"""Which form of a kernel a step takes, where the rule is Python's: steps of every make-up, without a GPU."""

from types import SimpleNamespace

import pytest
import torch

from miniserve_b200 import ops
from miniserve_b200.ops import mixers, native


@pytest.mark.parametrize("singles, others, chunks, head_chunks", [
    (0, [16], True, True), (0, [15], False, False), (0, [2048], True, True), (0, [1037, 640, 371], True, True),
    (0, [8, 8], False, True), (0, [2] * 64, False, True), (0, [4] * 64, False, True), (0, [16] * 64, True, True),
    (64, [16], False, True), (64, [64], False, True), (64, [512], True, True), (256, [512], True, True), (256, [511], False, True),
    (14, [2], False, True), (2, [2048, 1], True, True)])
def test_recurrences_by_chunks_where_rows_are_long_beside_the_decoding_ones(singles, others, chunks, head_chunks):
    """Decoding rows cost a chunk each: a short prompt beside many of them, or many rows of a few tokens, stays on the token-by-token walk."""
    t = singles + sum(others)
    ctx = SimpleNamespace(decode_only=False, num_rows=singles + len(others), leading_single_rows=singles)
    q = torch.empty(t, 64)
    assert mixers.walk_ok(q, q, q, 64, ctx) == chunks
    assert mixers.walk_ok(q, q, q, 64, ctx, head_decay=True) == head_chunks


@pytest.mark.parametrize("rows, keys, heads, dim, captured, tiled", [
    ([2], 2, 16, 128, False, False), ([2] * 16, 32, 16, 128, False, False), ([33], 33, 16, 128, False, True), ([40], 40, 4, 64, False, False),
    ([64], 64, 4, 64, False, False), ([65], 65, 4, 64, False, True), ([2], 4000, 4, 64, False, True), ([2], 2, 16, 128, True, True), ([1, 1], 4000, 16, 128, False, False)])
def test_32_bit_prompt_attention_in_tiles_where_there_is_more_than_a_tile_of_keys(monkeypatch, rows, keys, heads, dim, captured, tiled):
    monkeypatch.setattr(native, "kernels", lambda: SimpleNamespace(ms_attention_tiled_f32_supports=lambda *sizes: 1))
    ctx = SimpleNamespace(decode_only=all(n == 1 for n in rows), num_rows=len(rows), max_kv_len=keys, recorder=object() if captured else None)
    q, pool = torch.empty(sum(rows), heads, dim), torch.empty(1, heads, 16, dim)
    assert ops.attention_tiled_ok(torch.empty_like(q), q, pool, pool, ctx) == tiled
