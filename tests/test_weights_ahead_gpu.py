"""Kernels that ask for weights ahead of the wait on the kernel before them read everything else behind it: a captured chain whose kernels overlap
gives, for inputs that change from replay to replay, the bits of the same calls made one at a time."""
import pytest
import torch

from miniserve_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("ahead", [True, False])
@pytest.mark.parametrize("tokens, hidden, d", [(1, 1024, 128), (8, 1024, 128), (8, 2048, 128), (8, 2560, 128), (13, 1024, 256)])
def test_a_chain_of_overlapping_kernels(tokens, hidden, d, ahead):
    torch.manual_seed(tokens + hidden + d)
    nq, nkv, layers, page = 8, 4, 6, 16
    bf = dict(device=DEV, dtype=torch.bfloat16)
    i32 = dict(device=DEV, dtype=torch.int32)
    weights = [dict(qkv=torch.randn((nq + 2 * nkv) * d, hidden, **bf) / hidden ** 0.5, o=torch.randn(hidden, nq * d, **bf) / (nq * d) ** 0.5,
                    norm=torch.rand(hidden, **bf) + 0.5, q=torch.rand(d, **bf) + 0.5, k=torch.rand(d, **bf) + 0.5) for _ in range(layers)]
    inv_freq = 1e4 ** (-torch.arange(d // 2, device=DEV) / (d // 2))
    positions, rows = torch.zeros(tokens, **i32), torch.arange(tokens, **i32)
    indptr, pages, status = torch.arange(tokens + 1, **i32) * 4, torch.randperm(tokens * 4, device=DEV).int(), torch.zeros(1, **i32)
    x, residual, qkv = torch.empty(tokens, hidden, **bf), torch.empty(tokens, hidden, device=DEV), torch.empty(tokens, (nq + 2 * nkv) * d, **bf)
    q, delta = torch.empty(tokens, nq, d, **bf), torch.empty(tokens, hidden, **bf)
    k_pool, v_pool = (torch.zeros(layers, tokens * 4, nkv, page, d, **bf) for _ in range(2))

    def chain(stream, between=lambda: None):
        table = ops.rope_table(positions, inv_freq, tokens, d, stream=stream)
        between()
        for i, w in enumerate(weights):
            ops.linear(x, w["qkv"], out=qkv, stream=stream)
            between()
            ops.qk_norm_rope_kv(q, k_pool[i], v_pool[i], qkv, w["q"], w["k"], inv_freq, d, 1e-6, positions, rows, indptr, pages, page, status,
                                stream=stream, cos_sin=table, weights_ahead=ahead)
            between()
            ops.linear(q.view(tokens, nq * d), w["o"], out=delta, stream=stream)
            between()
            ops.add_rmsnorm(x, residual, delta, w["norm"], 1e-6, stream=stream, weights_ahead=ahead)
            between()

    def start(seed):
        gen = torch.Generator(device=DEV).manual_seed(seed)
        x.copy_(torch.randn(tokens, hidden, generator=gen, device=DEV))
        residual.copy_(torch.randn(tokens, hidden, generator=gen, device=DEV))
        positions.copy_(torch.randint(0, 4 * page, (tokens,), generator=gen, device=DEV))
        pages.copy_(torch.randperm(tokens * 4, generator=gen, device=DEV))
        k_pool.zero_()
        v_pool.zero_()

    def result():
        return [t.clone() for t in (x, residual, q, k_pool, v_pool)]

    start(0)
    chain(torch.cuda.current_stream().cuda_stream)  # (kernels are set up outside the capture)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain(torch.cuda.current_stream().cuda_stream)
    for seed in range(1, 5):
        start(seed)
        graph.replay()
        torch.cuda.synchronize()
        got = result()
        start(seed)
        torch.cuda.synchronize()
        chain(torch.cuda.current_stream().cuda_stream, torch.cuda.synchronize)
        for a, b in zip(got, result()):
            assert torch.equal(a, b)
    assert status.item() == 0


@pytest.mark.parametrize("hidden, d", [(1024, 128), (2048, 256)])
def test_weights_that_the_kernel_before_has_written(hidden, d):
    """Without ``weights_ahead`` a norm's weight may be what a kernel right before it writes, which lets its dependents start at once."""
    torch.manual_seed(hidden)
    k, tokens, nq, nkv, page = 8192, 4, 4, 2, 16
    bf, i32 = dict(device=DEV, dtype=torch.bfloat16), dict(device=DEV, dtype=torch.int32)
    make_norm, make_q = torch.randn(hidden, k, **bf) / k ** 0.5, torch.randn(d, k, **bf) / k ** 0.5
    residual, qkv, inv_freq = torch.randn(tokens, hidden, device=DEV), torch.randn(tokens, (nq + 2 * nkv) * d, **bf), torch.rand(d // 2, device=DEV)
    positions, rows, indptr, pages, status = torch.arange(tokens, **i32), torch.zeros(tokens, **i32), torch.tensor([0, 1], **i32), torch.zeros(1, **i32), torch.zeros(1, **i32)
    norm_w, q_w, k_w = torch.ones(1, hidden, **bf), torch.ones(1, d, **bf), torch.ones(1, d, **bf)
    out, q, kp, vp = torch.empty(tokens, hidden, **bf), torch.empty(tokens, nq, d, **bf), torch.zeros(1, nkv, page, d, **bf), torch.zeros(1, nkv, page, d, **bf)

    def run(x, between):
        ops.linear(x, make_norm, out=norm_w)
        between()
        ops.add_rmsnorm(out, residual, None, norm_w.view(-1), 1e-6, write_residual=False)
        ops.linear(x, make_q, out=q_w)
        ops.linear(x, make_q, out=k_w)
        between()
        ops.qk_norm_rope_kv(q, kp, vp, qkv, q_w.view(-1), k_w.view(-1), inv_freq, d, 1e-6, positions, rows, indptr, pages, page, status)
        torch.cuda.synchronize()
        return [t.clone() for t in (out, q, kp, vp)]

    for _ in range(4):
        x = torch.randn(1, k, **bf)
        for w in (norm_w, q_w, k_w):
            w.fill_(1.0)
        got = run(x, lambda: None)
        for a, b in zip(got, run(x, torch.cuda.synchronize)):
            assert torch.equal(a, b)
    assert status.item() == 0
