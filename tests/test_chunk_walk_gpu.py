"""The recurrences by chunks of 16 tokens (``csrc/chunk_walk.cu``) against the recurrence in 64-bit, beside the token-by-token walk on
the same operands: every rule, both types, odd sizes, rows from one token to several chunks, some behind an earlier state."""

from types import SimpleNamespace

import pytest
import torch

from miniserve_b200 import ops
from miniserve_b200.ops import mixers

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")
ROWS = [(0, 1), (5, 64), (0, 65), (300, 200), (0, 7), (9, 1), (0, 129), (64, 16), (0, 48)]
SLOTS = [6, 0, 3, 1, 4, 5, 2, 8, 7]


def _ctx(rows, slots):
    cu = [0]
    for _, n in rows:
        cu.append(cu[-1] + n)
    i32 = dict(dtype=torch.int32, device=DEV)
    held = {}
    return SimpleNamespace(
        cu_q=torch.tensor(cu, **i32), q_start=torch.tensor([s for s, _ in rows], **i32), state_slot=torch.tensor(slots, **i32),
        num_rows=len(rows), decode_only=False, held=held, stream=torch.cuda.current_stream().cuda_stream, step_cache={},
        buffer=lambda role, shape, dtype, dev: held.setdefault((role, shape, dtype), torch.empty(shape, dtype=dtype, device=dev)))


def _exact(q, k, v, decay, beta, rows, slots, held):
    """(outputs, the sizes of the terms that they are sums of, states behind) in 64-bit; q, k, decay [T, H, dk], v [T, H, dv], held
    [slots, H, dv, dk]."""
    out, size, last, t = [], [], held.clone(), 0
    for (start, n), slot in zip(rows, slots):
        s = held[slot].clone() if start else torch.zeros_like(held[slot])
        m = s.abs()  # the terms that s is a sum of, without their signs
        for _ in range(n):
            s, m = s * decay[t][:, None, :], m * decay[t][:, None, :]
            u = v[t] if beta is None else beta[t][:, None] * (v[t] - (s * k[t][:, None, :]).sum(-1))
            s, m = s + u[:, :, None] * k[t][:, None, :], m + (u[:, :, None] * k[t][:, None, :]).abs()
            out.append((s * q[t][:, None, :]).sum(-1))
            size.append((m * q[t].abs()[:, None, :]).sum(-1) + 1e-3)
            t += 1
        last[slot] = s
    return torch.stack(out), torch.stack(size), last


def _columns(gen, t, width, dtype, pad):
    """[T, width] as columns of wider rows that do not start at the row's beginning."""
    return torch.randn(t, width + 2 * pad, generator=gen).to(torch.bfloat16).to(dtype).to(DEV)[:, pad:pad + width]


ROUTES = {"chunks": dict(WALK_MIN_TOKENS=1), "walk": dict(WALK_MIN_TOKENS=1 << 30, SEGMENTS=1),
          "segments": dict(WALK_MIN_TOKENS=1 << 30, SEGMENT_MIN_TOKENS=1)}


def _by(route, run, q, k, v, dk, head_decay, rows, slots, state, heads, dv):
    """(outputs, the state behind) of one route."""
    kept = {name: getattr(mixers, name) for name in ROUTES[route]}
    try:
        for name, value in ROUTES[route].items():
            setattr(mixers, name, value)
        ctx = _ctx(rows, slots)
        assert mixers.walk_ok(q, k, v, dk, ctx, head_decay=head_decay) == (route == "chunks")
        st, o = state.clone(), torch.full((q.shape[0], heads, dv), float("nan"), device=DEV)
        run(o, st, ctx)
    finally:
        for name, value in kept.items():
            setattr(mixers, name, value)
    return o, st


def _both(run, q, k, v, dk, head_decay, want, size, last, state, heads, dv, delta=False):
    """By chunks, token by token, and (the decay rule) in segments: largest error over the terms' size, root mean square of it, of the states'."""
    errors = {}
    for route in ("chunks", "walk") if delta else ("chunks", "walk", "segments"):
        o, st = _by(route, run, q, k, v, dk, head_decay, ROWS, SLOTS, state, heads, dv)
        off, behind = (o.double().cpu() - want).abs() / size, (st.double().cpu() - last).abs()
        errors[route] = (off.max().item(), off.pow(2).mean().sqrt().item(), (behind.max() / last.abs().max()).item(), behind.pow(2).mean().sqrt().item())
    print(dk, dv, errors)
    # a float32 sum in any order: a few roundings of 6e-8 of the terms' sizes, at most one for each of them
    for route, e in errors.items():
        assert e[0] < 1e-6 and e[2] < 1e-6, (route, errors)
    # and chunks are no less accurate than the walk: two root mean squares over n numbers of like size differ by chance by 1 / sqrt(n) of
    # themselves, and these numbers' sizes differ
    for at, n in ((1, want.numel()), (3, last.numel())):
        assert errors["chunks"][at] < (1.05 + 10 / n ** 0.5) * errors["walk"][at], errors


@pytest.mark.parametrize("dtype, z_dtype", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16), (torch.float32, torch.bfloat16)])
@pytest.mark.parametrize("rule", ["decay", "delta"])
@pytest.mark.parametrize("heads, groups, dk, dv, pad", [(2, 1, 64, 64, 8), (3, 3, 10, 6, 3), (4, 2, 24, 40, 8), (1, 1, 72, 136, 1), (2, 2, 128, 16, 8),
                                                        (1, 1, 32, 17, 4), (1, 1, 1, 1, 0), (6, 2, 40, 20, 0)])
def test_channel_decays_by_chunks(dtype, z_dtype, rule, heads, groups, dk, dv, pad):
    gen = torch.Generator().manual_seed(dk * 1000 + dv)
    t, delta = sum(n for _, n in ROWS), rule == "delta"
    q, k = (_columns(gen, t, groups * dk, dtype, pad) for _ in range(2))
    if delta:  # unit keys, as the layer makes them
        k = (k.float().view(t, groups, dk) / k.float().view(t, groups, dk).norm(dim=-1, keepdim=True)).view(t, -1).to(dtype)
    v = _columns(gen, t, heads * dv, dtype, pad)
    z = torch.randn(t, heads * dk, generator=gen) * 2
    z[::17] = 60.0       # sign +1: a decay that is next to nothing, again and again
    z[3::29] = -60.0     # a decay of one
    z[70:90] = 20.0      # nothing is left, for several tokens in a row
    z = z.to(z_dtype).to(DEV)
    bias, coef = (torch.randn(heads * dk, generator=gen) * 0.3).to(DEV), (torch.rand(heads, generator=gen) + 0.2).to(DEV)
    beta = torch.randn(t, heads + 3, generator=gen).to(z_dtype).to(DEV)[:, 2:2 + heads] if delta else None
    scale = torch.rand(t, heads, generator=gen).to(DEV) if pad == 0 else None  # (a factor per token and head on the values)
    state = torch.randn(len(ROWS), heads, dv, dk, generator=gen).to(DEV)
    vd = v.double().cpu().view(t, heads, dv) * (1.0 if scale is None else scale.double().cpu()[:, :, None])
    wide = lambda x: x.double().cpu().view(t, groups, dk).repeat_interleave(heads // groups, dim=1)  # noqa: E731
    soft = torch.nn.functional.softplus(z.double().cpu() + bias.double().cpu(), threshold=1e9).view(t, heads, dk)
    decay = torch.exp(-coef.double().cpu()[None, :, None] * soft)
    exact = _exact(wide(q) * 0.3, wide(k), vd, decay, torch.sigmoid(beta.double().cpu()) if delta else None,
                   ROWS, SLOTS, state.double().cpu())
    _both(lambda o, st, ctx: ops.decay_scan(o, st, q, k, v, z, bias, coef, 1.0, beta, ctx, heads, dk, dv, 0.3, delta=delta,
                                            v_scale=scale),
          q, k, v, dk, False, *exact, state, heads, dv, delta)


@pytest.mark.parametrize("rule, heads, dk, dv, exact", [("decay", 2, 136, 24, False), ("delta", 2, 136, 24, False), ("delta", 1, 256, 6, False),
                                                        ("decay", 2, 24, 40, True), ("delta", 3, 64, 20, True)])
def test_prompts_that_stay_on_the_walk(rule, heads, dk, dv, exact):
    """More than 128 key channels, and what 32-bit models ask for: token by token over prompts (the decay rule of 531 tokens in segments)."""
    gen = torch.Generator().manual_seed(dk)
    t = sum(n for _, n in ROWS)
    q, k, v = torch.randn(t, heads * dk, generator=gen).to(DEV), torch.randn(t, heads, dk, generator=gen), torch.randn(t, heads * dv, generator=gen).to(DEV)
    k = (k / k.norm(dim=-1, keepdim=True)).reshape(t, -1).to(DEV)
    z, bias, coef = torch.randn(t, heads * dk, generator=gen).to(DEV), torch.zeros(heads * dk, device=DEV), torch.ones(heads, device=DEV)
    beta = torch.randn(t, heads, generator=gen).to(DEV) if rule == "delta" else None
    state, ctx = torch.randn(len(ROWS), heads, dv, dk, generator=gen).to(DEV), _ctx(ROWS, SLOTS)
    wide = lambda x: x.double().cpu().view(t, heads, -1)  # noqa: E731
    decay = torch.exp(-torch.nn.functional.softplus(wide(z)))
    want, size, last = _exact(wide(q) * 0.25, wide(k), wide(v), decay, None if beta is None else torch.sigmoid(beta.double().cpu()), ROWS, SLOTS,
                              state.double().cpu())
    assert exact or not mixers.walk_ok(q, k, v, dk, ctx)
    o, st = torch.full((t, heads, dv), float("nan"), device=DEV), state.clone()
    ops.decay_scan(o, st, q, k, v, z, bias, coef, 1.0, beta, ctx, heads, dk, dv, 0.25, delta=rule == "delta", exact=exact)
    assert not any(role.startswith("walk") for role, *_ in ctx.held)
    assert ((o.double().cpu() - want).abs() / size).max() < 1e-6 and ((st.double().cpu() - last).abs().max() / last.abs().max()) < 1e-6


@pytest.mark.parametrize("heads, groups, dk, dv, scaled", [(8, 2, 128, 64, True), (4, 4, 64, 16, True), (2, 1, 32, 33, False), (160, 2, 32, 70, True),
                                                           (40, 1, 128, 1, False)])
def test_head_decays_by_chunks(heads, groups, dk, dv, scaled):
    gen = torch.Generator().manual_seed(heads)
    t = sum(n for _, n in ROWS)
    q, k = (torch.randn(t, groups * dk + 8, generator=gen).to(DEV)[:, 4:4 + groups * dk] for _ in range(2))
    v = torch.randn(t, heads * dv + 1, generator=gen).to(DEV)[:, 1:]
    a = torch.rand(t, heads, generator=gen)
    a[::13], a[5::19], a[70:90] = 0.0, 1.0, 1e-20
    a = a.to(DEV)
    scale = torch.rand(t, heads, generator=gen).to(DEV) if scaled else None
    state = torch.randn(len(ROWS), heads, dv, dk, generator=gen).to(DEV)
    wide = lambda x: x.double().cpu().reshape(t, groups, dk).repeat_interleave(heads // groups, dim=1)  # noqa: E731
    vd = v.double().cpu().reshape(t, heads, dv) * (scale.double().cpu()[:, :, None] if scaled else 1.0)
    exact = _exact(wide(q) * 0.7, wide(k), vd, a.double().cpu()[:, :, None].expand(t, heads, dk), None, ROWS, SLOTS, state.double().cpu())
    _both(lambda o, st, ctx: ops.decay_scan(o, st, q, k, v, a, None, None, 0.0, None, ctx, heads, dk, dv, 0.7, delta=False, head_decay=True,
                                            v_scale=scale), q, k, v, dk, True, *exact, state, heads, dv)


def test_many_rows():
    """More rows than a warp has lanes, empty ones among them (also the first and the last)."""
    gen = torch.Generator().manual_seed(7)
    lens = [0, 1, 16, 17, 0, 0, 33] * 11 + [1] * 70 + [50, 0]
    rows, slots = [(3 * (i % 2), n) for i, n in enumerate(lens)], torch.randperm(len(lens), generator=gen).tolist()
    t, heads, d = sum(lens), 2, 32
    q, k, v = (torch.randn(t, heads * d, generator=gen).to(DEV) for _ in range(3))
    a, state = torch.rand(t, heads, generator=gen).to(DEV), torch.randn(len(rows), heads, d, d, generator=gen).to(DEV)
    wide = lambda x: x.double().cpu().view(t, heads, d)  # noqa: E731
    want, size, last = _exact(wide(q), wide(k), wide(v), a.double().cpu()[:, :, None].expand(t, heads, d), None, rows, slots, state.double().cpu())
    for (start, n), slot in zip(rows, slots):
        if n == 0:  # an empty row is no step of its request
            last[slot] = state[slot].double().cpu()
    ctx = _ctx(rows, slots)
    o, st = torch.full((t, heads, d), float("nan"), device=DEV), state.clone()
    ops.decay_scan(o, st, q, k, v, a, None, None, 0.0, None, ctx, heads, d, d, 1.0, delta=False, head_decay=True)
    assert ((o.double().cpu() - want).abs() / size).max() < 1e-6 and ((st.double().cpu() - last).abs().max() / last.abs().max()) < 4e-6


def _operands(rule, gen, t, heads, dk, dv, lo, hi):
    """Operands whose decays are uniform in [lo, hi], and how to run them: (run, q, k, v, exact decays, beta, factor on the values)."""
    rnd, uni = (lambda *s: torch.randn(*s, generator=gen).to(DEV)), (lambda *s: torch.rand(*s, generator=gen).to(DEV))
    q, k, v = rnd(t, heads * dk), rnd(t, heads, dk), rnd(t, heads * dv)
    k = (k / k.norm(dim=-1, keepdim=True)).reshape(t, -1).contiguous()
    if rule == "head":
        a, scale = lo + (hi - lo) * uni(t, heads), uni(t, heads) * 0.1 + 0.01
        return (lambda o, st, ctx: ops.decay_scan(o, st, q, k, v, a, None, None, 0.0, None, ctx, heads, dk, dv, 0.25, delta=False, head_decay=True,
                                                  v_scale=scale)), q, k, v, a.double().cpu()[:, :, None].expand(t, heads, dk), None, scale, a
    coef, bias = uni(heads) * 0.5 + 0.2, torch.zeros(heads * dk, device=DEV)
    decay = (lo + (hi - lo) * uni(t, heads * dk).double()).clamp(max=1 - 2.0 ** -22)
    z = torch.log(torch.expm1(-torch.log(decay) / coef.double().repeat_interleave(dk))).float()
    soft = torch.nn.functional.softplus(z.double().cpu(), threshold=1e9)
    exact = torch.exp(-coef.double().cpu().repeat_interleave(dk) * soft).view(t, heads, dk)
    beta = rnd(t, heads) if rule == "delta" else None
    return (lambda o, st, ctx: ops.decay_scan(o, st, q, k, v, z, bias, coef, 1.0, beta, ctx, heads, dk, dv, 0.25, delta=rule == "delta")), \
        q, k, v, exact, None if beta is None else torch.sigmoid(beta.double().cpu()), None, z


@pytest.mark.parametrize("rule, heads, dk, dv", [("decay", 2, 64, 64), ("delta", 2, 64, 64), ("head", 2, 128, 64)])
@pytest.mark.parametrize("lo, hi", [(0.02, 0.6), (0.7, 0.99), (0.999, 1.0), (0.9999, 1.0)])
def test_long_rows_by_chunks_are_as_accurate_as_the_walk(rule, heads, dk, dv, lo, hi):
    """2,048 tokens behind a stored state: states of a token or two, and states that last from the first token to the last."""
    gen = torch.Generator().manual_seed(int(hi * 100) + dk)
    rows, slots, t = [(9, 2048), (0, 40)], [1, 0], 2088
    run, q, k, v, decay, beta, scale, _ = _operands(rule, gen, t, heads, dk, dv, lo, hi)
    state = torch.randn(2, heads, dv, dk, generator=gen).to(DEV)
    wide = lambda x: x.double().cpu().view(t, heads, -1)  # noqa: E731
    vd = wide(v) * (1.0 if scale is None else scale.double().cpu()[:, :, None])
    want, _, last = _exact(wide(q) * 0.25, wide(k), vd, decay, beta, rows, slots, state.double().cpu())
    errors = {}
    for route in ("chunks", "walk"):
        o, st = _by(route, run, q, k, v, dk, rule == "head", rows, slots, state, heads, dv)
        off, behind = o.double().cpu() - want, (st.double().cpu() - last) / last.pow(2).mean().sqrt()
        errors[route] = (off.pow(2).mean().sqrt() / want.pow(2).mean().sqrt()).item(), behind.pow(2).mean().sqrt().item()
    print(rule, lo, hi, errors)
    assert all(c < 1.05 * w for c, w in zip(errors["chunks"], errors["walk"])), errors


@pytest.mark.parametrize("rule, heads, dk, dv", [("decay", 2, 64, 24), ("delta", 2, 40, 64), ("head", 2, 32, 33)])
@pytest.mark.parametrize("where, bad", [(w, float(b)) for w in ("v", "k", "q", "state") for b in ("inf", "nan")]
                         + [("decay", float("nan")), ("v", -3.4e38), ("state", -1e37)])
def test_values_that_are_not_finite_stay_with_their_token_and_the_later_ones(rule, heads, dk, dv, where, bad):
    """The same outputs and states are finite as token by token (also beside numbers near the largest), the others what they are without."""
    gen = torch.Generator().manual_seed(3)
    rows, slots, t = [(4, 37), (0, 20)], [1, 0], 57
    run, q, k, v, _, _, _, z = _operands(rule, gen, t, heads, dk, dv, 0.7, 0.99)
    state = torch.randn(2, heads, dv, dk, generator=gen).to(DEV)
    args = q, k, v, dk, rule == "head", rows, slots
    plain = _by("chunks", run, *args, state, heads, dv)
    if where == "state":
        state[1, 0, 3, 5] = bad
    else:
        dict(v=v, k=k, q=q, decay=z)[where][21, 1] = bad
    got, want = (_by(route, run, *args, state, heads, dv) for route in ("chunks", "walk"))
    for g, w, p in zip(got, want, plain):
        assert torch.equal(torch.isfinite(g), torch.isfinite(w))
        own = (w - p).abs() <= 1e-5 * p.abs().max()  # (what the number does not reach; the walk says which)
        assert own.float().mean() > 0.5 and ((g - p).abs()[own] <= 2e-5 * p.abs().max()).all()


@pytest.mark.parametrize("kind", ["decay", "delta", "state_space"])
def test_cuts_change_no_bit_of_a_32_bit_layer(kind):
    """The 32-bit mode stays on the token-by-token walk: the same bits however a prompt is cut into portions, and whatever comes with it."""
    from miniserve_b200.config import PartSpec
    from miniserve_b200.parts import BuildEnv, build_part
    from tests import test_fekulix_gpu as fekulix
    from tests import test_rofozen_gpu as rofozen

    torch.manual_seed(5)
    if kind == "state_space":
        part, _ = rofozen._ssm(torch.float32, 4, 16, 32, 2, 4, 2)
        rofozen._bind(part, torch.float32, change=rofozen._ssm_weights)
    else:
        names = dict(q="q", k="k", v="v", g="g", o="o", norm="norm", a1="a1", a2="a2", a_bias="a2.b")
        spec = PartSpec("decay_linear_attention", dict(hidden=48, heads=2, key_dim=24, value_dim=40, tau=5.0, decay_rank=8, eps=1e-5, names=names))
        if kind == "delta":
            spec = PartSpec("gated_delta_rule", dict(
                hidden=48, heads=4, kv_heads=2, key_dim=16, value_dim=24, conv=3, decay_rank=8, gate_rank=16, eps=1e-5,
                names=dict(q="q", k="k", v="v", q_conv="q.conv", k_conv="k.conv", v_conv="v.conv", beta="b", a_log="A_log", norm="norm", a1="a1",
                           a2="a2", dt_bias="dt_bias", g1="g1", g2="g2", o="o")))
        part = build_part("mixer", spec, BuildEnv(torch.float32, DEV))
        fekulix._bind(part, torch.float32)
    width = rofozen.HIDDEN if kind == "state_space" else 48
    views, x = fekulix._state_views(part), torch.randn(60, width, device=DEV)
    whole = fekulix._portions(part, views, x, (60,), 1, torch.float32)
    for cuts in ((20, 3, 37), (15, 15, 15, 15), (44, 16)):
        assert torch.equal(fekulix._portions(part, views, x, cuts, 1, torch.float32), whole), cuts
