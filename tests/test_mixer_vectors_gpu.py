"""The four-channels-a-thread forms of the convolution, the per-head norm and the grouped norm against the forms for any operand, which
the same numbers take when their rows do not start on whole vectors: sizes around the edges of a thread, a warp and a run of tokens."""

from types import SimpleNamespace

import pytest
import torch

from miniserve_b200 import ops

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")


def _rows(lens, started):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    i32 = dict(dtype=torch.int32, device=DEV)
    return SimpleNamespace(cu_q=torch.tensor(cu, **i32), q_start=torch.tensor(started, **i32), state_slot=torch.arange(len(lens) - 1, -1, -1, **i32),
                           row_of_token=torch.tensor([r for r, n in enumerate(lens) for _ in range(n)], **i32), num_rows=len(lens),
                           stream=torch.cuda.current_stream().cuda_stream)


def _view(gen, t, width, ahead, dtype):
    """[T, width] behind ``ahead`` columns of rows as wide as whole fours allow (ahead odd: no whole vectors)."""
    full = torch.randn(t, -(-(width + ahead) // 4) * 4 + 4, generator=gen).to(dtype).to(DEV)
    return full[:, ahead:ahead + width]


def _near(a, b, dtype):
    # the two forms add a norm's squares in other orders: a few units in the last place of float32, then one rounding
    tol = 2e-6 if dtype == torch.float32 else 2.0 ** -7
    assert not torch.isnan(b).any() and ((a.float() - b.float()).abs() <= tol * b.float().abs() + 1e-6).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("taps, unit, dk, others, dv", [(4, 4, 64, 5, 36), (3, 2, 16, 3, 8), (2, 1, 128, 1, 4), (4, 0, 1, 6, 700), (2, 3, 4, 2, 6)])
@pytest.mark.parametrize("lens, started", [((1, 1, 1), (0, 3, 1)), ((5, 1, 8, 700, 2, 3), (0, 9, 2, 1, 0, 5)), ((2048,), (0,))])
def test_convolution_in_fours(dtype, taps, unit, dk, others, dv, lens, started):
    gen = torch.Generator().manual_seed(taps * 100 + unit)
    ctx, t, c = _rows(lens, started), sum(lens), unit * dk + others * dv
    x = _view(gen, t, c, 4, dtype)
    odd = torch.empty(t, c + 7, dtype=dtype, device=DEV)[:, 1:1 + c]
    odd.copy_(x)
    state = torch.randn(len(lens), taps - 1, c, generator=gen).to(dtype).to(DEV)
    w, bias = torch.randn(c, taps, generator=gen).to(DEV), torch.randn(c, generator=gen).to(DEV)
    got, want = (torch.full((t, c), float("nan"), device=DEV) for _ in range(2))
    for b in (None, bias):
        ops.conv_silu_unit(got, x, state, w, ctx, unit, dk, others, dv, 1e-6, bias=b)
        ops.conv_silu_unit(want, odd, state, w, ctx, unit, dk, others, dv, 1e-6, bias=b)
        _near(got, want, torch.float32)
    # the histories behind the step, made with the outputs (in one launch where every row has one token) and by the launch for any rows
    left = state.clone()
    ops.conv_state_update(left, x, ctx, taps)
    ctx.decode_only = max(lens) == 1
    for operand in (x, odd):
        moved = state.clone()
        ops.conv_silu_unit(want, operand, moved, w, ctx, unit, dk, others, dv, 1e-6, bias=bias, update=True)
        assert torch.equal(moved, left)
        _near(got, want, torch.float32)


@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("lens", [(1, 1), (301, 9)])
def test_convolution_with_taps_at_any_address(taps, lens):
    """Four channels' taps are read as whole vectors where they are aligned: the same bits where they are not."""
    gen = torch.Generator().manual_seed(taps)
    ctx, t, c = _rows(lens, (0, 5)), sum(lens), 2052
    x, state = torch.randn(t, c, generator=gen).bfloat16().to(DEV), torch.randn(len(lens), taps - 1, c, generator=gen).bfloat16().to(DEV)
    w = torch.randn(c, taps, generator=gen).to(DEV)
    moved = torch.empty(c * taps + 1, device=DEV)[1:].view(c, taps).copy_(w)
    assert w.data_ptr() % 16 == 0 and moved.data_ptr() % 16 == 4
    got, want = (torch.full((t, c), float("nan"), device=DEV) for _ in range(2))
    ops.conv_silu_unit(got, x, state, w, ctx, 0, 1, c // 4, 4, 1e-6)
    ops.conv_silu_unit(want, x, state, moved, ctx, 0, 1, c // 4, 4, 1e-6)
    assert not torch.isnan(got).any() and torch.equal(got, want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("t, heads, dv", [(1, 1, 64), (37, 3, 32), (130, 5, 128), (3, 7, 64)])
@pytest.mark.parametrize("kind, own", [("silu", False), ("sigmoid", True)])
def test_head_norm_in_fours(dtype, t, heads, dv, kind, own):
    gen = torch.Generator().manual_seed(t + dv)
    o, w = torch.randn(t, heads, dv, generator=gen).to(DEV), torch.randn(heads * dv if own else dv, generator=gen).to(DEV)
    gate = _view(gen, t, heads * dv, 4, dtype)
    odd = torch.empty(t, heads * dv + 3, dtype=dtype, device=DEV)[:, 1:1 + heads * dv]
    odd.copy_(gate)
    got, want = (torch.full((t, heads * dv), float("nan"), dtype=dtype, device=DEV) for _ in range(2))
    ops.head_norm_gate(got, o, w, gate, 1e-5, 0.7, kind)
    ops.head_norm_gate(want, o, w, odd, 1e-5, 0.7, kind)
    _near(got, want, dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("t, parts, size, dv, skip", [(1, 1, 4, 4, True), (9, 8, 512, 64, True), (5, 3, 260, 52, False), (3, 2, 1024, 128, True),
                                                      (2, 1, 252, 12, True), (500, 1, 1024, 64, True), (460, 1, 260, 52, False)])
def test_group_norm_in_fours(dtype, t, parts, size, dv, skip):
    gen = torch.Generator().manual_seed(size)
    width = parts * size
    o, w = torch.randn(t, width, generator=gen).to(DEV), torch.randn(width, generator=gen).to(DEV)
    x = _view(gen, t, width, 4, torch.float32) if skip else None
    s = torch.randn(width // dv, generator=gen).to(DEV) if skip else None
    gate = _view(gen, t, width, 4, dtype)
    odd = torch.empty(t, width + 3, dtype=dtype, device=DEV)[:, 1:1 + width]
    odd.copy_(gate)
    got, want = (torch.full((t, width), float("nan"), dtype=dtype, device=DEV) for _ in range(2))
    ops.gated_group_norm(got, o, x, s, gate, w, parts, dv, 1e-6)
    ops.gated_group_norm(want, o, x, s, odd, w, parts, dv, 1e-6)
    _near(got, want, dtype)


@pytest.mark.parametrize("size, parts", [(512, 2), (1024, 1), (64, 4)])
def test_float32_norms_of_a_token_are_the_same_bits_in_any_step(size, parts):
    """One token, a few and many: what the step holds beside a token picks no other order of its sums."""
    gen = torch.Generator().manual_seed(size)
    t, width = 600, size * parts
    o, gate, w = (torch.randn(*s, generator=gen).to(DEV) for s in ((t, width), (t, width), (width,)))
    whole = torch.empty(t, width, device=DEV)
    ops.gated_group_norm(whole, o, None, None, gate, w, parts, 32, 1e-6)
    for n in (1, 7, 150):
        part = torch.empty(n, width, device=DEV)
        ops.gated_group_norm(part, o[:n].contiguous(), None, None, gate[:n].contiguous(), w, parts, 32, 1e-6)
        assert torch.equal(part, whole[:n])


@pytest.mark.parametrize("c, unit, dk", [(96, 1, 32), (2048, 16, 64)])
def test_float32_convolutions_of_a_token_are_the_same_bits_in_any_step(c, unit, dk):
    gen = torch.Generator().manual_seed(c)
    t = 800
    x, w, state = torch.randn(t, c, generator=gen).to(DEV), torch.randn(c, 4, generator=gen).to(DEV), torch.zeros(1, 3, c, device=DEV)
    outs = []
    for n in (t, 201, 40, 1):
        out = torch.empty(n, c, device=DEV)
        ops.conv_silu_unit(out, x[:n], state, w, _rows((n,), (0,)), unit, dk, c // dk - unit, dk, 1e-6)
        outs.append(out)
    assert all(torch.equal(o, outs[0][:o.shape[0]]) for o in outs)


def _held(ctx, decode):
    kept = {}
    ctx.decode_only, ctx.step_cache = decode, {}
    ctx.buffer = lambda role, shape, dtype, dev: kept.setdefault((role, shape, dtype), torch.empty(shape, dtype=dtype, device=dev))
    return ctx


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads, dv, n, groups, taps, parts", [(4, 32, 64, 2, 4, 2), (6, 20, 20, 3, 1, 1), (3, 7, 32, 1, 3, 1), (8, 64, 128, 8, 2, 4), (2, 6, 18, 1, 4, 1)])
@pytest.mark.parametrize("lens, started", [((1, 1, 1), (0, 3, 1)), ((5, 1, 8, 40), (0, 9, 2, 1)), ((3, 2), (1, 0))])
def test_state_space_features_in_one_call(dtype, heads, dv, n, groups, taps, parts, lens, started):
    """The one native call against the single ones, bit for bit, and only for the steps that it takes."""
    gen = torch.Generator().manual_seed(heads + taps)
    t, inner, decode = sum(lens), heads * dv, all(k == 1 for k in lens)
    c = inner + 2 * groups * n
    proj = torch.randn(t, -(-(inner + c + heads) // 8) * 8, generator=gen).to(dtype).to(DEV)
    f = lambda *shape: torch.randn(*shape, generator=gen).to(DEV)  # noqa: E731
    w_conv, conv_bias, dt_bias, coef, skip, norm = f(c, taps), f(c), f(heads), f(heads).exp(), f(heads), f(inner)
    state, conv = f(len(lens), heads, dv, n), f(len(lens), taps - 1, c).to(dtype)
    unit = max(u for u in range(1, 129) if c % u == 0)
    ctx = _held(_rows(lens, started), decode)
    ctx.leading_single_rows, ctx.sm_count = next((i for i, k in enumerate(lens) if k != 1), len(lens)), 148
    exact = dtype == torch.float32
    out = torch.full((t, inner), float("nan"), dtype=dtype, device=DEV)
    got_state, got_conv = state.clone(), conv.clone()
    taken = ops.ssm_features(out, proj, got_state, got_conv if taps > 1 else None, w_conv, conv_bias, dt_bias, coef, skip, norm, ctx, heads, dv, n, groups, unit,
                             parts, 1e-6, exact)
    assert taken == ((decode and n % 4 == 0) or (not decode and not exact and t >= 16 and n in (32, 64, 128) and inner % 4 == 0))
    if not taken:
        assert torch.equal(got_state, state) and torch.equal(got_conv, conv)
        return
    xbc, steps, o, want = f(t, c), f(2, t, heads), f(t, heads, dv), torch.full((t, inner), float("nan"), dtype=dtype, device=DEV)
    ops.conv_silu_unit(xbc, proj[:, inner:inner + c], conv, w_conv, ctx, 0, 1, c // unit, unit, 0.0, bias=conv_bias, update=taps > 1)
    ops.ssm_step_decay(steps, proj[:, inner + c:inner + c + heads], dt_bias, coef)
    xs, bs, cs = torch.split_with_sizes(xbc, (inner, groups * n, groups * n), 1)
    ops.decay_scan(o, state, cs, bs, xs, steps[1], None, coef, 1.0, None, ctx, heads, n, dv, 1.0, delta=False, head_decay=True, v_scale=steps[0], exact=exact)
    ops.gated_group_norm(want, o.view(t, inner), xs, skip, proj[:, :inner], norm, parts, dv, 1e-6)
    assert torch.equal(out, want) and torch.equal(got_state, state) and torch.equal(got_conv, conv)


@pytest.mark.parametrize("t, hidden, inter, experts, extra, top, kind", [(1, 64, 40, 5, 1, 2, "gated"), (9, 72, 64, 12, 0, 3, "clamped"), (300, 64, 48, 4, 2, 2, "plain"),
                                                                        (40, 128, 136, 3, 1, 1, "shared")])
def test_routed_feed_forward_in_one_call(t, hidden, inter, experts, extra, top, kind):
    from miniserve_b200.ops import experts as xo

    gen = torch.Generator().manual_seed(t)
    f = lambda *shape: torch.randn(*shape, generator=gen).to(DEV)  # noqa: E731
    r, gated = experts + extra, kind != "plain"
    x, router, correction = f(t, hidden).bfloat16(), f(r, hidden) * hidden ** -0.5, f(r) * 0.01
    w_up, w_down = (f(experts, (2 if gated else 1) * inter, hidden) * hidden ** -0.5).bfloat16(), (f(experts, hidden, inter) * inter ** -0.5).bfloat16()
    clamps = (2.0, 1.7, 1.0) if kind == "clamped" else None
    shared, gate_w = (f(t, hidden).bfloat16(), f(hidden)) if kind == "shared" else (None, None)
    gates = [None if gate_w is None else torch.empty(t, device=DEV) for _ in range(2)]
    ctx = _held(_rows((t,), (0,)), False)
    got = xo.experts_forward(x, ctx, router, correction, None, gate_w, gates[0], w_up, w_down, shared, top, 1, 1, 1, 1.5, True, "softmax", False, 0.0, gated,
                             not gated, clamps)
    slots, i32 = t * top, dict(dtype=torch.int32, device=DEV)
    rows = xo.tc_tile_rows(slots, experts)
    idx, wgt, pos, perm, offsets = torch.empty(t, top, **i32), f(t, top), torch.empty(slots, **i32), torch.empty(slots, **i32), torch.empty(experts + 1, **i32)
    tiles, meta = torch.empty(xo.expert_max_tiles(slots, experts, rows), 2, **i32), torch.empty(2, **i32)
    xs, act, y, want = torch.zeros(slots, hidden, dtype=x.dtype, device=DEV), torch.empty(slots, inter, dtype=x.dtype, device=DEV), f(slots, hidden), torch.empty_like(x)
    xo.expert_route(idx, wgt, x, router, correction, top, 1, 1, 1.5, True, gate_w=gate_w, gate_out=gates[1])
    xo.expert_plan(pos, perm, offsets, tiles, meta, idx, experts, tile_rows=rows)
    xo.expert_gather(xs, x, perm, meta, top)
    xo.expert_products_tc(act, xs, w_up, tiles, meta, offsets, gated, relu_squared=not gated, clamps=clamps, tile_rows=rows)
    xo.expert_products_tc(y, act, w_down, tiles, meta, offsets, False, tile_rows=rows)
    xo.expert_combine(want, y, x, idx, wgt, pos, experts, shared=shared, shared_gate=gates[1])
    torch.cuda.synchronize()
    assert torch.equal(got, want) and ops.device_status("cuda").item() == 0 and (gate_w is None or torch.equal(*gates))
