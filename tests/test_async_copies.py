"""Asynchronous copies into shared memory are written so that the compiler moves no access of shared memory across them."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "miniserve_b200" / "csrc"


@pytest.mark.parametrize("source", ["chunk_mma.cuh", "chunk_walk.cu", "attention_rowwise.cu"])
def test_copies_and_waits_name_memory(source):
    """A wait that is not followed by a barrier is all that keeps the loads behind it in place."""
    text = (CSRC / source).read_text()
    statements = [s for s in re.findall(r"asm volatile\((?:.|\n)*?\);", text) if "cp.async" in s]
    assert statements
    for s in statements:
        assert re.search(r':\s*"memory"\s*\);$', s), s
