"""The plan of routed experts: a counting sort of slots by expert, and the tiles of its rows."""
import pytest
import torch

from miniserve_b200 import ops  # noqa: F401  (loads the kernels)
from miniserve_b200.ops import native

pytestmark = pytest.mark.gpu
DEV = "cuda"


# 16 slots a thread stay in registers (16,384); experts are added up 32 at a time
@pytest.mark.parametrize("slots", [1, 1023, 1025, 16384, 16385, 40000])
@pytest.mark.parametrize("experts, tile", [(1, 64), (31, 64), (33, 1), (64, 128), (1500, 7)])
def test_plan(slots, experts, tile):
    gen = torch.Generator(device=DEV).manual_seed(slots + experts)
    idx = torch.randint(0, experts + 2, (slots,), generator=gen, device=DEV, dtype=torch.int32)  # (from `experts` on: identity)
    if experts > 2:
        idx[idx == 1] = 2  # an expert that nobody uses
    k = native.experts()
    most = k.ms_expert_max_tiles_of(slots, experts, tile)
    pos, perm = (torch.full((slots,), -7, device=DEV, dtype=torch.int32) for _ in range(2))
    offsets = torch.full((experts + 1,), -7, device=DEV, dtype=torch.int32)
    tiles, meta = torch.full((most, 2), -7, device=DEV, dtype=torch.int32), torch.empty(2, device=DEV, dtype=torch.int32)
    assert k.ms_expert_plan_of(pos.data_ptr(), perm.data_ptr(), offsets.data_ptr(), tiles.data_ptr(), meta.data_ptr(), idx.data_ptr(), slots, experts,
                               tile, torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    ids = idx.tolist()
    counts = [0] * experts
    for e in ids:
        if e < experts:
            counts[e] += 1
    begin, want_tiles = [0], []
    for e, n in enumerate(counts):
        want_tiles += [[e, begin[-1] + r] for r in range(0, n, tile)]
        begin.append(begin[-1] + n)
    assert offsets.tolist() == begin and meta.tolist() == [len(want_tiles), begin[-1]] and tiles.tolist()[:len(want_tiles)] == want_tiles
    where, back = pos.tolist(), perm.tolist()
    for slot, e in enumerate(ids):
        if e >= experts:
            assert where[slot] == -1
        else:
            assert begin[e] <= where[slot] < begin[e + 1] and back[where[slot]] == slot
