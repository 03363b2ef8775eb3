"""The decay rule over long rows by chunks of 64 tokens on the tensor cores (``csrc/tile_walk.cu``) against the recurrence in 64-bit, beside
the token-by-token walk on the same operands: edges of chunks, sixteens, column tiles and segments, odd sizes, values that are not finite."""

import pytest
import torch

from miniserve_b200 import ops
from miniserve_b200.ops import mixers, native
from tests.test_chunk_walk_gpu import DEV, _columns, _ctx, _exact, _operands

pytestmark = pytest.mark.gpu


def _run(run, route, rows, slots, state, q, heads, dv):
    kept = mixers.WALK_MIN_TOKENS, mixers.SEGMENTS
    try:
        if route == "walk":
            mixers.WALK_MIN_TOKENS, mixers.SEGMENTS = 1 << 30, 1
        st, o = state.clone(), torch.full((q.shape[0], heads, dv), float("nan"), device=DEV)
        run(o, st, _ctx(rows, slots))
    finally:
        mixers.WALK_MIN_TOKENS, mixers.SEGMENTS = kept
    return o, st


def _takes(rows, heads, dk, dv, groups):
    return native.recurrence().ms_walk_kernels(sum(n for _, n in rows), len(rows), heads, dk, dv, 0, groups) == 3


def _compare(run, rows, slots, q, want, size, last, state, heads, dv):
    errors = {}
    for route in ("tiles", "walk"):
        o, st = _run(run, route, rows, slots, state, q, heads, dv)
        off, behind = (o.double().cpu() - want).abs() / size, (st.double().cpu() - last).abs()
        errors[route] = (off.max().item(), off.pow(2).mean().sqrt().item(), (behind.max() / last.abs().max()).item(), behind.pow(2).mean().sqrt().item())
    print(errors)
    for e in errors.values():  # a few roundings of 6e-8 of the terms' sizes
        assert e[0] < 1e-6 and e[2] < 1e-6, errors
    for at, n in ((1, want.numel()), (3, last.numel())):  # and no further off than token by token (two root mean squares over n numbers)
        assert errors["tiles"][at] < (1.05 + 10 / n ** 0.5) * errors["walk"][at], errors
    assert ops.device_status(DEV).item() == 0


@pytest.mark.parametrize("heads, groups, dk, dv, pad, dtype", [(2, 1, 64, 64, 8, torch.bfloat16), (3, 3, 10, 6, 3, torch.float32), (1, 1, 72, 136, 1, torch.bfloat16),
                                                               (2, 2, 128, 17, 0, torch.float32), (80, 2, 24, 70, 4, torch.bfloat16)])
def test_channel_decays(heads, groups, dk, dv, pad, dtype):
    gen = torch.Generator().manual_seed(dk)
    rows, slots = [(5, 1225), (0, 65)], [1, 0]
    assert _takes(rows, heads, dk, dv, 0)
    t = 1290
    q, k = (_columns(gen, t, groups * dk, dtype, pad) for _ in range(2))
    v = _columns(gen, t, heads * dv, dtype, pad)
    z = torch.randn(t, heads * dk, generator=gen) * 2
    z[::17], z[3::29], z[70:90] = 60.0, -60.0, 20.0
    z = z.to(dtype).to(DEV)
    bias, coef = (torch.randn(heads * dk, generator=gen) * 0.3).to(DEV), (torch.rand(heads, generator=gen) + 0.2).to(DEV)
    scale = torch.rand(t, heads, generator=gen).to(DEV) if pad == 0 else None
    state = torch.randn(2, heads, dv, dk, generator=gen).to(DEV)
    vd = v.double().cpu().view(t, heads, dv) * (1.0 if scale is None else scale.double().cpu()[:, :, None])
    wide = lambda x: x.double().cpu().view(t, groups, dk).repeat_interleave(heads // groups, dim=1)  # noqa: E731
    soft = torch.nn.functional.softplus(z.double().cpu() + bias.double().cpu(), threshold=1e9).view(t, heads, dk)
    exact = _exact(wide(q) * 0.3, wide(k), vd, torch.exp(-coef.double().cpu()[None, :, None] * soft), None, rows, slots, state.double().cpu())
    _compare(lambda o, st, ctx: ops.decay_scan(o, st, q, k, v, z, bias, coef, 1.0, None, ctx, heads, dk, dv, 0.3, delta=False, v_scale=scale), rows, slots, q, *exact,
             state, heads, dv)


@pytest.mark.parametrize("heads, groups, dk, dv, scaled", [(8, 2, 128, 64, True), (4, 4, 64, 16, True), (2, 1, 32, 33, False), (160, 2, 32, 70, True)])
def test_head_decays(heads, groups, dk, dv, scaled):
    gen = torch.Generator().manual_seed(heads)
    rows, slots = [(5, 401), (0, 65), (300, 128), (0, 1)], [3, 0, 1, 2]
    assert _takes(rows, heads, dk, dv, groups)
    t = sum(n for _, n in rows)
    q, k = (torch.randn(t, groups * dk + 8, generator=gen).to(DEV)[:, 4:4 + groups * dk] for _ in range(2))
    v = torch.randn(t, heads * dv + 1, generator=gen).to(DEV)[:, 1:]
    a = torch.rand(t, heads, generator=gen)
    a[::13], a[5::19], a[70:90] = 0.0, 1.0, 1e-20
    a = a.to(DEV)
    scale = torch.rand(t, heads, generator=gen).to(DEV) if scaled else None
    state = torch.randn(len(rows), heads, dv, dk, generator=gen).to(DEV)
    wide = lambda x: x.double().cpu().reshape(t, groups, dk).repeat_interleave(heads // groups, dim=1)  # noqa: E731
    vd = v.double().cpu().reshape(t, heads, dv) * (scale.double().cpu()[:, :, None] if scaled else 1.0)
    exact = _exact(wide(q) * 0.7, wide(k), vd, a.double().cpu()[:, :, None].expand(t, heads, dk), None, rows, slots, state.double().cpu())
    _compare(lambda o, st, ctx: ops.decay_scan(o, st, q, k, v, a, None, None, 0.0, None, ctx, heads, dk, dv, 0.7, delta=False, head_decay=True, v_scale=scale),
             rows, slots, q, *exact, state, heads, dv)


def _spread(where, gen, q, k, v, state):
    """[T, H, d] operands and [1, H, dv, dk] states with numbers far larger than the others, in place."""
    if where == "a value channel":
        v[:, :, 5] *= 1024
    elif where == "a key channel":
        k[:, :, 5] *= 1024
        state[..., 5] *= 1024
    elif where == "a query channel":
        q[:, :, 5] *= 1024
    elif where == "tokens":
        k[::97] *= 1024
        v[40::97] *= 4096
    elif where == "some values":
        v[torch.rand(v.shape, generator=gen, device=DEV) < 0.01] *= 16384
    elif where == "keys against queries":  # the products are as large as without
        by = torch.exp2(torch.randint(-12, 13, (k.shape[2],), generator=gen, device=DEV).float())
        k *= by
        q /= by
        state *= by
    else:
        assert where == "everything"
        for x in (q, k, v, state):
            x *= torch.exp2(4 * torch.randn(x.shape, generator=gen, device=DEV))


@pytest.mark.parametrize("rule, heads, dk, dv, t", [("decay", 3, 64, 72, 1301), ("decay", 2, 128, 64, 1301), ("head", 3, 128, 64, 431), ("head", 2, 32, 40, 431)])
@pytest.mark.parametrize("low, high", [(0.02, 0.6), (0.9, 0.999), (0.9999, 0.99999)])
@pytest.mark.parametrize("where", ["a value channel", "a key channel", "a query channel", "tokens", "some values", "keys against queries", "everything"])
def test_numbers_of_very_different_sizes(rule, heads, dk, dv, t, low, high, where):
    """The error of every output and of every number of the state against the size of its own terms: a large number takes no bits from others."""
    gen = torch.Generator(device=DEV).manual_seed(dk + dv)
    q, k, v, state = (torch.randn(s, generator=gen, device=DEV) for s in ((t, heads, dk), (t, heads, dk), (t, heads, dv), (1, heads, dv, dk)))
    _spread(where, gen, q, k, v, state)
    a = low + (high - low) * torch.rand(t, heads, dk if rule == "decay" else 1, generator=gen, device=DEV)
    rows, st, o, flat = [(7, t)], state.clone(), torch.empty(t, heads, dv, device=DEV), [x.reshape(t, -1) for x in (q, k, v)]
    assert _takes(rows, heads, dk, dv, heads if rule == "head" else 0)
    if rule == "head":
        ops.decay_scan(o, st, *flat, a.reshape(t, heads), None, None, 0.0, None, _ctx(rows, [0]), heads, dk, dv, 1.0, delta=False, head_decay=True)
        a = a.double()
    else:
        z = torch.log(torch.expm1(-torch.log(a.double()))).float()
        ops.decay_scan(o, st, *flat, z.reshape(t, -1), torch.zeros(heads * dk, device=DEV), torch.ones(heads, device=DEV), 1.0, None, _ctx(rows, [0]), heads, dk, dv,
                       1.0, delta=False)
        a = torch.exp(-torch.nn.functional.softplus(z.double(), threshold=1e9))
    q, k, v, exact = q.double(), k.double(), v.double(), state[0].double()
    size = exact.abs()
    worst = torch.zeros((), dtype=torch.float64, device=DEV)
    for i in range(t):
        u = v[i][:, :, None] * k[i][:, None, :]
        exact, size = exact * a[i][:, None, :] + u, size * a[i][:, None, :] + u.abs()
        off = (o[i].double() - (exact * q[i][:, None, :]).sum(-1)).abs() / (size * q[i].abs()[:, None, :]).sum(-1)
        worst = torch.maximum(worst, off.max())
    behind = ((st[0].double() - exact).abs() / size).max().item()
    # At most eight cuts of 2^-23 of a sum no larger than its terms' (9.5e-7), hardly ever one after the other. Decays made of logits come on top: each is
    # off by up to 2^-24 (expf's last bit, below one), and as many of them are in a term as it has been kept for, on average no more than 1 / (1 - decay) tokens.
    most = 1e-6 + (rule == "decay") * min(t, 1 / (1 - (low + high) / 2)) * 2.0 ** -24
    assert worst.item() < most and behind < most, (worst.item(), behind)
    assert ops.device_status(DEV).item() == 0


@pytest.mark.parametrize("rule, dk, dv, n", [("decay", 64, 128, 1300), ("head", 128, 64, 1000)])
def test_heads_that_fill_the_gpu_walk_rows_whole(rule, dk, dv, n):
    """Few heads: rows in segments. The same bits beside so many heads that rows stay whole, behind a state and from zero."""
    gen = torch.Generator().manual_seed(1)
    many, few, rows = 160, 2, [(7, n)]
    run, q, k, v, _, _, scale, z = _operands(rule, gen, n, many, dk, dv, 0.7, 0.999)
    state = torch.randn(1, many, dv, dk, generator=gen).to(DEV)
    coef = torch.ones(many, device=DEV)

    def go(heads, start):
        ctx, st, o = _ctx([(start, n)], [0]), state[:, :heads].clone(), torch.empty(n, heads, dv, device=DEV)
        cut = lambda x, d: x[:, :heads * d]  # noqa: E731
        if rule == "head":
            ops.decay_scan(o, st, cut(q, dk), cut(k, dk), cut(v, dv), z[:, :heads].contiguous(), None, None, 0.0, None, ctx, heads, dk, dv, 0.25, delta=False,
                           head_decay=True, v_scale=scale[:, :heads].contiguous())
        else:
            ops.decay_scan(o, st, cut(q, dk), cut(k, dk), cut(v, dv), cut(z, dk), torch.zeros(heads * dk, device=DEV), coef[:heads], 1.0, None, ctx, heads, dk, dv, 0.25,
                           delta=False)
        return o, st

    assert _takes(rows, few, dk, dv, few if rule == "head" else 0)
    for start in (7, 0):
        (o, st), (oo, so) = go(few, start), go(many, start)
        assert torch.equal(o, oo[:, :few]) and torch.equal(st, so[:, :few])


@pytest.mark.parametrize("rule, heads, dk, dv, rows", [("decay", 2, 64, 24, [(4, 1300), (0, 20)]), ("head", 2, 32, 33, [(4, 437), (0, 20)])])
@pytest.mark.parametrize("where, bad", [(w, float(b)) for w in ("v", "k", "q", "state") for b in ("inf", "nan")] + [("decay", float("nan")), ("v", -3.4e38), ("state", -1e37)])
def test_values_that_are_not_finite_stay_with_their_token_and_the_later_ones(rule, heads, dk, dv, rows, where, bad):
    gen = torch.Generator().manual_seed(3)
    slots, t = [1, 0], sum(n for _, n in rows)
    run, q, k, v, _, _, _, z = _operands(rule, gen, t, heads, dk, dv, 0.7, 0.99)
    assert _takes(rows, heads, dk, dv, heads if rule == "head" else 0)
    state = torch.randn(2, heads, dv, dk, generator=gen).to(DEV)
    plain = _run(run, "tiles", rows, slots, state, q, heads, dv)
    if where == "state":
        state[1, 0, 3, 5] = bad
    else:
        dict(v=v, k=k, q=q, decay=z)[where][121, 1] = bad
    got, want = (_run(run, route, rows, slots, state, q, heads, dv) for route in ("tiles", "walk"))
    for g, w, p in zip(got, want, plain):
        assert torch.equal(torch.isfinite(g), torch.isfinite(w))
        own = (w - p).abs() <= 1e-5 * p.abs().max()  # (what the number does not reach; the walk says which)
        assert own.float().mean() > 0.5 and ((g - p).abs()[own] <= 2e-5 * p.abs().max()).all()


@pytest.mark.parametrize("dk", [64, 128])
@pytest.mark.parametrize("no_queries, no_added", [(0, 1 << 30), (2, 1 << 30), (1 << 30, 0), (1 << 30, 3), (1, 1)])
def test_copies_that_do_not_come_end_the_walk_with_an_error(dk, no_queries, no_added):
    """The walk ends by itself with the status word raised, whichever of its roles waits in vain; a state that lacks what a chunk adds is not kept."""
    gen = torch.Generator().manual_seed(1)
    heads, dv, rows = 2, 64, [(4, 300), (0, 400)]
    t, lib, ctx = sum(n for _, n in rows), native.recurrence(), _ctx(rows, [1, 0])
    q, k, v = (torch.randn(t, heads * d, generator=gen).to(DEV) for d in (dk, dk, dv))
    decay, state = torch.rand(t, heads, generator=gen).to(DEV), torch.randn(2, heads, dv, dk, generator=gen).to(DEV)
    scratch = torch.zeros(lib.ms_tile_walk_scratch(t, len(rows), heads, dk, dv, heads), device=DEV)

    def go(none_q, none_added):
        o, st, status = torch.zeros(t, heads, dv, device=DEV), state.clone(), torch.zeros(1, dtype=torch.int32, device=DEV)
        native.recurrence_check(lib.ms_tile_walk_selftest(o.data_ptr(), st.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), decay.data_ptr(),
                                                          scratch.data_ptr(), ctx.cu_q.data_ptr(), ctx.q_start.data_ptr(), ctx.state_slot.data_ptr(), t, len(rows), heads,
                                                          dk, dv, status.data_ptr(), none_q, none_added, 20_000_000, ctx.stream), launches=3)
        torch.cuda.synchronize()
        return o, st, status.item()

    want = go(1 << 30, 1 << 30)
    assert want[2] == 0 and torch.isfinite(want[0]).all() and not torch.equal(want[1], state)
    _, st, status = go(no_queries, no_added)
    assert status == 42
    if no_added < 4:  # both rows have five chunks or more
        assert torch.equal(st, state)
    again = go(1 << 30, 1 << 30)
    assert torch.equal(again[0], want[0]) and torch.equal(again[1], want[1]) and again[2] == 0


# us by chunks of 64 and of 16 on a B200: (heads, dk, dv), groups (0: a decay per channel), tokens, rows
@pytest.mark.parametrize("shape, groups, tokens, rows, tiles", [
    ((32, 128, 128), 0, 2048, 1, True),    # 274, 324
    ((32, 128, 128), 0, 300, 1, False),    # 69, 53
    ((16, 128, 128), 0, 512, 1, False),    # 54, 52
    ((8, 64, 128), 0, 2048, 1, True),      # 65, 91
    ((8, 64, 128), 0, 640, 1, False),      # 36, 34
    ((16, 128, 64), 0, 640, 1, False),     # 65, 51
    ((64, 64, 64), 0, 640, 1, False),      # 94, 83
    ((64, 128, 128), 0, 512, 1, True),     # 147, 165
    ((4, 64, 64), 0, 900, 1, True),        # 32, 41
    ((64, 32, 32), 0, 2048, 1, False),     # 243, 174
    ((64, 128, 64), 8, 300, 1, True),      # 42, 48
    ((64, 128, 64), 8, 2048, 3, True),     # 160, 254
    ((4, 64, 64), 1, 300, 1, False),       # 21, 18
    ((16, 64, 64), 2, 400, 1, False),      # 25, 22
    ((16, 64, 64), 2, 512, 1, True),       # 26, 26
])
def test_which_steps_go_by_chunks_of_64(shape, groups, tokens, rows, tiles):
    assert (native.recurrence().ms_walk_kernels(tokens, rows, *shape, 0, groups) == 3) == tiles
