"""bfloat16 tensor-core attention (``csrc/attention_bf16.cu``), compiled per head size on first
use: a model only pays for the head size it has."""

from __future__ import annotations

import ctypes
from ctypes import c_char_p, c_float, c_int, c_longlong, c_void_p
from functools import lru_cache

import torch

import miniserve_b200.ops as ops

from . import build, native

_p, _i, _f, _ll = c_void_p, c_int, c_float, c_longlong


def _flag(name: str, default: str) -> bool:
    import os

    return os.environ.get(name, default) == "1"


CLUSTER_MERGE = _flag("MINISERVE_CLUSTER_MERGE", "1")  # 2 to 8 key splits of a decode step as one thread-block cluster


def supports(head_dim: int, page_size: int) -> bool:
    return head_dim % 16 == 0 and 16 <= head_dim <= 256 and page_size & (page_size - 1) == 0


def takes_extras(head_dim: int, page_size: int) -> bool:
    """Whether these kernels take learned sink scores, a cap on the scores, a mask by blocks of positions, a distance
    bias and kept first keys."""
    return supports(head_dim, page_size)


_NO_EXTRAS = (None, 0.0, 0, None, None, 0)


def _extras_args(extras) -> tuple:
    if extras is None:
        return _NO_EXTRAS
    sv, r1, r2 = extras.sink_values, extras.dist_r1, extras.dist_r2
    return (None if sv is None else sv.data_ptr(), float(extras.softcap or 0.0), int(extras.chunk or 0),
            None if r1 is None else r1.data_ptr(), None if r2 is None else r2.data_ptr(), int(extras.keep_first or 0))


def module_for(head_dim: int) -> build.Module:
    return build.Module(f"attn_bf16_d{head_dim}", ("attention_bf16.cu",), defines=(f"MS_HEAD_DIM={head_dim}",))


@lru_cache(maxsize=None)
def _lib(head_dim: int):
    if not supports(head_dim, 16):
        raise ValueError(f"the bfloat16 attention kernels take head sizes that are multiples of 16 up to 256, not {head_dim}")
    lib = ctypes.CDLL(str(build.ensure_built(module_for(head_dim))))
    pre = f"ms_attn_bf16_d{head_dim}_"
    fns = {}
    for name, args, res in (
        ("last_error", [], c_char_p),
        ("prefill", [_p] * 8 + [_i, _i, _i, _i, _f, _i, _i, _i, _p, _p, _f, _i, _p, _p, _i], c_int),
        ("decode", [_p] * 9 + [_i, _i, _i, _f, _i, _i, _i, _i, _p], c_int),
        ("decode_fused", [_p] * 10 + [_i, _i, _i, _f, _i, _i, _i, _i, _p, _p, _f, _i, _p, _p, _i, _ll, _p, _i], c_int),
        ("decode_cluster", [_p] * 7 + [_i, _i, _i, _f, _i, _i, _i, _i, _p, _p, _f, _i, _p, _p, _i, _ll, _p], c_int),
        ("decode_clusters_resident", [_i, _i, ctypes.POINTER(c_int)], c_int),
    ):
        fn = getattr(lib, pre + name)
        fn.argtypes, fn.restype = args, res
        fns[name] = fn
    set_pdl = getattr(lib, pre + "set_pdl")
    set_pdl.argtypes, set_pdl.restype = [c_int], None
    set_pdl(int(native.pdl_enabled()))
    fns["lib"] = lib
    return fns


def _check(fns, rc: int, launches: int = 1) -> None:
    native.LAUNCHES[0] += launches
    if rc != 0:
        raise native.NativeError(fns["last_error"]().decode())


@lru_cache(maxsize=None)
def clusters_resident(head_dim: int, splits: int, device_index: int = 0, copies: bool = True) -> int:
    """How many thread-block clusters of ``splits`` decode CTAs the device holds at a time (a cluster
    lies within one GPC: on a B200 with head size 128, 71 clusters of 4 and 33 of 8, not 74 and 37). ``copies``: of the form that
    brings its slices by tensor copies (``takes_tensor_copies``), else of the general one."""
    fns = _lib(head_dim)
    out = c_int(0)
    with torch.cuda.device(device_index):
        rc = fns["decode_clusters_resident"](splits, int(copies), ctypes.byref(out))
    if rc != 0:
        raise native.NativeError(fns["last_error"]().decode())
    return out.value


def choose_splits(rows: int, head_chunks: int, max_kv_len: int | None, sm_count: int, resident=None) -> int:
    """How many ways the keys of each (request, kv head) are split across CTAs: as many as give
    one wave of two CTAs per SM, but at least 128 keys per split and at most 16 splits up to 4,096 keys
    (measured on B200 at contexts of 512 to 4,096 and batches of 1 to 32: more splits only add partial
    results to merge, fewer leave SMs idle; one split too many and the CTAs no longer fit one wave: a
    decode step of 8 requests at 2,048 tokens takes 1.28 ms with 4 splits, 1.34 with 3, 1.60 with 8).
    Beyond that a split is not asked to walk more than 256 keys while CTAs would be idle: a single
    request of 8,192 keys is cut 32 ways, of 32,768 keys 37 ways (every CTA that fits): 1.33 -> 1.15 ms
    per step at 8,192 keys, 2.83 -> 1.60 at 32,768, 9.01 -> 3.43 at 131,072 (4.7 TB/s).
    ``max_kv_len`` None (inside a CUDA graph for short contexts, where the launch cannot follow the
    context length): assume a few thousand keys, and stay within the 8 splits that one thread-block
    cluster merges (a single request: 0.98 ms per step with 8 splits, 0.99 with 16).
    ``resident(splits)``: how many clusters of that size the device holds at a time; splits that run
    as a cluster (2 to 8) are reduced until every (request, head group) has its cluster in the first
    wave (6 requests x 8 head groups in clusters of 6: 48 clusters where 45 fit, and the step took 1.33 ms
    against 1.17 for 8 requests in clusters of 4). A few more than 8 splits are not worth leaving the
    cluster for: 9 to 11 become 8."""
    items = max(rows * head_chunks, 1)
    want = (2 * sm_count) // items
    by_len = 8 if max_kv_len is None else max(1, -(-max_kv_len // 128))
    most = 16 if max_kv_len is None else max(16, max_kv_len // 256)
    splits = max(1, min(want, by_len, most))
    if 8 < splits < 12:
        splits = 8
    if resident is not None:
        while 2 <= splits <= 8 and resident(splits) < items:
            splits -= 1
    return splits


def takes_tensor_copies(rows: int, splits: int, head_dim: int, page_size: int) -> bool:
    """Whether a decode launch brings its slices of keys by tensor copies (head sizes 64 and 128, pages that hold whole slices of 16).
    A few rows stay with the copies of 16 bytes a lane: their warps have a few slices each, of which the first comes sooner that way
    (us, tensor copies against those: 1 row of 300 keys 4.84 / 4.47, of 2,048 8.72 / 8.38, 2 of 2,048 9.71 / 9.36, 4 of 300 5.34 / 5.07;
    from 8 rows on the other way round: 8 of 300 6.08 / 6.34, of 2,048 16.9 / 17.4, of 8,192 46.6 / 49.9, 64 of 2,048 86 / 93), unless
    several long rows are cut many ways (2 of 8,192 19.9 / 20.4, of 32,768 51.5 / 53.0). One row takes the same alone (of 8,192 14.9 / 14.9,
    of 32,768 32.7 / 33.0, of 131,072 97.8 / 102); of its decode step, where the kernels before hide the other form's start, 8,192 keys
    1,153 / 1,148, 32,768 1,610 / 1,597, 65,536 2,184 / 2,222, 131,072 3,385 / 3,496: the general form up to the commoner lengths."""
    return head_dim in (64, 128) and page_size >= 16 and (rows >= 8 or (rows >= 2 and splits > 16))


@lru_cache(maxsize=None)
def _status_at(device_index: int) -> int:
    """The address of the device's status word, which lives as long as the process."""
    return ops.device_status(torch.device("cuda", device_index)).data_ptr()


def _scratch(ctx, need: int, d: int, device) -> tuple[torch.Tensor, torch.Tensor]:
    """Partial results: ``need`` rows of d floats, and of two."""
    if ctx.graph_bucket:
        # inside a CUDA graph capture: memory of the graph's own pool, alive as long as the graph
        return (torch.empty(need * d, dtype=torch.float32, device=device),
                torch.empty(need * 2, dtype=torch.float32, device=device))
    buf = ctx.scratch.get("attn_decode")
    if buf is None or buf[0].numel() < need * d or buf[1].numel() < need * 2:
        buf = (torch.empty(need * d, dtype=torch.float32, device=device),
               torch.empty(need * 2, dtype=torch.float32, device=device))
        ctx.scratch["attn_decode"] = buf
    return buf


def _counters(ctx, items: int, device) -> torch.Tensor:
    """Tickets of the merges inside the kernels: zero before the first launch, left zero by every launch."""
    counters = ctx.scratch.get("attn_counters")
    if counters is None or counters.numel() < items:
        if counters is not None:  # captured graphs may hold the smaller one's address: it stays alive
            ctx.scratch.setdefault("retired", []).append(counters)
        counters = torch.zeros(max(4096, items), dtype=torch.int32, device=device)
        ctx.scratch["attn_counters"] = counters
    return counters


def run(out: torch.Tensor, q: torch.Tensor, k_pool: torch.Tensor, v_pool: torch.Tensor, ctx, group: int,
        scale: float, window: int | None, sink: bool = False, extras=None) -> None:
    """The step's attention: rows at the front that bring one token each go to the split-key
    decode kernel, the rest to the tiled kernel."""
    single = ctx.leading_single_rows
    if single:
        run_decode(out, q, k_pool, v_pool, ctx, group, scale, window, single, sink, extras)
    if single < ctx.num_rows:
        run_prefill(out, q, k_pool, v_pool, ctx, group, scale, window, single, sink, extras)


def run_decode(out: torch.Tensor, q: torch.Tensor, k_pool: torch.Tensor, v_pool: torch.Tensor, ctx, group: int,
               scale: float, window: int | None, rows: int, sink: bool = False, extras=None, form: str | None = None) -> None:
    """Rows [0, rows) of the step, one new token each (so token i belongs to row i): keys split
    across CTAs, partial results merged by the last CTA of each (row, head group) to finish. ``form`` (tests):
    "general", copies of 16 bytes a lane, as head sizes other than 64 and 128 and pages of 8 tokens take."""
    t, nq, d = q.shape
    pages, nkv, page_size, _ = k_pool.shape
    fns = _lib(d)
    indptr, indices = ctx.page_indptr[group], ctx.page_indices[group]
    chunks = nkv * -(-(nq // nkv) // 16)
    fit = None
    if CLUSTER_MERGE:
        fit = lambda n: clusters_resident(d, n, q.device.index or 0, form != "general" and takes_tensor_copies(rows, n, d, page_size))  # noqa: E731
    known = ctx.max_kv_len if not ctx.graph_bucket else (getattr(ctx, "graph_kv_len", 0) or None)
    splits = choose_splits(rows, chunks, known, ctx.sm_count, fit)
    pool = (0, None)
    if rows > 1 and takes_tensor_copies(rows, splits, d, page_size) and form != "general":
        pool = (pages, _status_at(q.device.index))
    if CLUSTER_MERGE and 2 <= splits <= 8:
        # the splits as one thread-block cluster: merged through distributed shared memory
        _check(fns, fns["decode_cluster"](
            out.data_ptr(), q.data_ptr(), k_pool.data_ptr(), v_pool.data_ptr(), ctx.kv_len.data_ptr(), indptr.data_ptr(),
            indices.data_ptr(), rows, nq, nkv, float(scale), int(window or 0), int(sink), page_size, splits, ctx.stream,
            *_extras_args(extras), *pool))
        return
    merge = (None, None, None)
    if splits > 1:
        part_o, part_ml = _scratch(ctx, rows * nq * splits, d, q.device)
        counters = _counters(ctx, rows * chunks, q.device)
        merge = (part_o.data_ptr(), part_ml.data_ptr(), counters.data_ptr())
    _check(fns, fns["decode_fused"](
        out.data_ptr(), *merge, q.data_ptr(), k_pool.data_ptr(), v_pool.data_ptr(), ctx.kv_len.data_ptr(), indptr.data_ptr(),
        indices.data_ptr(), rows, nq, nkv, float(scale), int(window or 0), int(sink), page_size, splits, ctx.stream,
        *_extras_args(extras), *pool, int(known or 0)))


def run_prefill(out: torch.Tensor, q: torch.Tensor, k_pool: torch.Tensor, v_pool: torch.Tensor, ctx, group: int,
                scale: float, window: int | None, first_row: int = 0, sink: bool = False, extras=None) -> None:
    """Rows [first_row, num_rows) of the step, any number of new tokens each: tiles of 64 queries
    over the row's pages (``mma.sync``; the tcgen05 kernel of ``attention_tc.cu`` takes head size 128)."""
    t, nq, d = q.shape
    nkv, page_size = k_pool.shape[1], k_pool.shape[2]
    fns = _lib(d)
    indptr, indices = ctx.page_indptr[group], ctx.page_indices[group]
    skip = 4 * first_row  # the per-row tables are int32
    _check(fns, fns["prefill"](
        out.data_ptr(), q.data_ptr(), k_pool.data_ptr(), v_pool.data_ptr(), ctx.cu_q.data_ptr() + skip, ctx.q_start.data_ptr() + skip,
        indptr.data_ptr() + skip, indices.data_ptr(), ctx.num_rows - first_row, ctx.max_q_len, nq, nkv, float(scale), int(window or 0),
        int(sink), page_size, ctx.stream, *_extras_args(extras)))
