"""Kernels that may start while the ones before them still run read what those write through pointers made behind the wait (``csrc/common.cuh``): the compiler may load
through a `const __restrict__` parameter ahead of it. Looked up in the sources: every such parameter goes through ``pdl_prologue`` or ``pdl_wait``, or is read by
loads that stay where they stand."""
import re
from pathlib import Path

import pytest

SOURCES = sorted((Path(__file__).resolve().parent.parent / "miniserve_b200" / "csrc").glob("*.cu"))
# Read ahead of the wait on purpose, or by copies in assembly: weights of products, a decode step's older keys and values and its metadata.
AHEAD = {"gemm_skinny_kernel": {"W"}, "gemm_skinny_stream_kernel": {"W"}, "qk_norm_rope_kv_bf16_token_kernel": {"q_norm_w", "k_norm_w"},
         "attn_decode_kernel": {"k_pool", "v_pool", "kv_len_ptr", "page_indptr", "page_indices"}}
# Read through pointers made of them, whose loads are all written out: (the parameter, what is made of it)
MADE = {"gemm_f32_tiled_kernel": {"A": "ap", "W": "wp"}, "attn_prefill_tc_kernel": {"page_indices": "pages"}}
# Handed on to functions that read them by loads that are written out
HANDED_ON = {"attn_prefill_tc_kernel": ({"cu_q", "q_start"}, {"at_tile", "at_order", "at_claim"})}


def _closing(text, at, left, right):
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == left) - (text[i] == right)
        if depth == 0:
            return i
    raise AssertionError("no end")


def kernels(text):
    """(name, parameters, body) of every kernel."""
    for m in re.finditer(r"__global__", text):
        at = m.end()
        while True:
            opening = text.index("(", at)
            if not text[at:opening].rstrip().endswith("__launch_bounds__"):
                break
            at = _closing(text, opening, "(", ")") + 1
        name = re.search(r"(\w+)\s*$", text[at:opening]).group(1)
        end = _closing(text, opening, "(", ")")
        begin = text.index("{", end)
        params, depth, part = [], 0, ""
        for ch in text[opening + 1:end] + ",":
            depth += (ch in "<(") - (ch in ">)")
            if ch == "," and depth == 0:
                params.append(part)
                part = ""
            else:
                part += ch
        yield name, params, text[begin:_closing(text, begin, "{", "}")]


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_pointers_go_through_the_wait(path):
    text = re.sub(r"//[^\n]*", "", path.read_text())
    for name, params, body in kernels(text):
        waits = re.findall(r"pdl_(?:prologue|wait)\(([^)]*)\)", body)
        if not waits:
            continue  # launched behind everything before it
        passed = {p.strip() for w in waits for p in w.split(",")}
        read_only = {re.search(r"(\w+)\s*$", p).group(1) for p in params if re.search(r"\bconst\b.*__restrict__", p)}
        for pointer, made in MADE.get(name, {}).items():
            assert not re.search(r"reinterpret_cast<[^>]*>\(%s\b|\*%s\b" % (made, made), body.replace("*" + made + "[LA]", "").replace("*" + made + "[LW]", ""))
            assert made + "[" not in body.replace(made + "[LA]", "").replace(made + "[LW]", "").replace(made + "[i]", "")
            passed.add(pointer)
        pointers, functions = HANDED_ON.get(name, ((), ()))
        for function in functions:
            begin = text.index("{", _closing(text, text.index(function + "("), "(", ")"))
            assert not re.search(r"\b(%s)\[" % "|".join(pointers), text[begin:_closing(text, begin, "{", "}")]), function
        passed |= set(pointers)
        for pointer in read_only - passed - AHEAD.get(name, set()):
            rest = re.sub(r"behind_(?:load\w*|four)\(\s*%s\b|\b%s != nullptr|if \(%s\)" % (pointer, pointer, pointer), "", body)
            rest = re.sub(r"threadIdx\.x|\b[a-z]\w*(?:\[i\])?\.[xyzw]\b", "", rest)
            uses = [u for u in re.findall(r"[^;{}]*\b%s\b[^;{}]*" % pointer, rest) if not re.fullmatch(r"\s*(?:if \([^;]*\) )?%s \+= [^;]*" % pointer, u)]
            assert not uses, (name, pointer, uses)
