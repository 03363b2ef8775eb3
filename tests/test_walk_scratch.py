"""What the walks over long rows ask for beside their operands: the cache pool leaves room for their scratch, and a plan belongs to one device."""
from types import SimpleNamespace

import torch

from miniserve_b200.engine.engine import Engine
from miniserve_b200.ops import mixers, native
from miniserve_b200.parts.base import FixedState, PagedKV
from miniserve_b200.parts.decoder import EntryCache

HEADS, WIDTH, STEP, RUNNING = 32, 128, 8192, 4


def _left(monkeypatch, need):
    """Bytes that are left beside pool and states of a device with 20 GB free, all of which the pool may take."""
    free = 20 << 30
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda device: (free, free))
    paged = PagedKV(kv_heads=8, head_dim=128)
    model = SimpleNamespace(dtype=torch.bfloat16, device="cuda:0", entry_caches=[EntryCache(0, (paged, need) if need else paged)],
                            spec=SimpleNamespace(hidden_size=64, vocab_size=1000))
    pages, = Engine._pool_pages(model, None, 16, 1.0, STEP, RUNNING)
    states = RUNNING * 4 * HEADS * WIDTH * WIDTH if need else 0
    return free - pages * 2 * 8 * 128 * 2 * 16 - states


def test_the_pool_leaves_room_for_the_walks_scratch(monkeypatch):
    dense, recurrent = _left(monkeypatch, None), _left(monkeypatch, FixedState((HEADS, WIDTH, WIDTH)))
    most = 4 << 28  # (a step whose scratch would be more stays on the chunks of 16)
    assert recurrent - dense >= most - (1 << 20)  # (pages are whole)
    assert dense < 3 << 29  # (and a model without such layers gives up nothing)


def test_a_plan_belongs_to_one_device(monkeypatch):
    asked = []

    def plan(*sizes):
        asked.append(sizes)
        return len(asked)

    monkeypatch.setattr(native, "recurrence", lambda: SimpleNamespace(ms_walk_scratch=plan, ms_walk_kernels=plan))
    mixers._walk_plan.cache_clear()
    sizes = (2048, 1, HEADS, WIDTH, WIDTH, False, 0)
    first, second = mixers._walk_plan(0, *sizes), mixers._walk_plan(1, *sizes)
    assert first != second and mixers._walk_plan(0, *sizes) == first and len(asked) == 4
    mixers._walk_plan.cache_clear()
