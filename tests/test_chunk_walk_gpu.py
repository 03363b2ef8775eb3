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
        num_rows=len(rows), decode_only=False, stream=torch.cuda.current_stream().cuda_stream, step_cache={},
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


def _both(run, q, k, v, dk, head_decay, want, size, last, state, heads, dv):
    """Runs by chunks and token by token: (largest error over the terms' size, its root mean square, the states' largest error) of each."""
    errors = {}
    for name, least in (("chunks", 1), ("walk", 1 << 30)):
        kept, mixers.WALK_MIN_TOKENS = mixers.WALK_MIN_TOKENS, least
        try:
            ctx = _ctx(ROWS, SLOTS)
            assert mixers.walk_ok(q, k, v, dk, ctx, head_decay=head_decay) == (name == "chunks")
            st, o = state.clone(), torch.full((q.shape[0], heads, dv), float("nan"), device=DEV)
            run(o, st, ctx)
        finally:
            mixers.WALK_MIN_TOKENS = kept
        off = (o.double().cpu() - want).abs() / size
        errors[name] = (off.max().item(), off.pow(2).mean().sqrt().item(), ((st.double().cpu() - last).abs().max() / last.abs().max()).item())
    print(dk, dv, errors)
    # factors of 22 bits (2.4e-7 a product) and float32 sums: below 1e-6 of the terms' sizes
    assert errors["chunks"][0] < 1e-6 and errors["chunks"][2] < 4e-6, errors


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
          q, k, v, dk, False, *exact, state, heads, dv)


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
