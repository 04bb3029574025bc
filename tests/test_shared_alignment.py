"""Shared arrays that are filled or read 16 bytes at a time declare that
alignment: without it their place follows from what else the kernel holds."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mtt-gpu-solver_b200", "csrc")
WIDE = [re.compile(r"\bcopy(?:_async)?16\(\s*&?(\w+)"),
        re.compile(r"reinterpret_cast<\s*(?:const\s+)?(?:u?int4|float4)\s*\*\s*>\(\s*&?(\w+)")]


def _shared(text):
    """Name -> whether its declaration is aligned to 16 bytes or more."""
    out = {}
    for line in re.findall(r"^[^\n;/]*__shared__[^;]*;", text, re.M):
        ok = any(int(n) >= 16 for n in re.findall(r"(?:__align__|alignas)\((\d+)\)", line))
        body = re.sub(r"(?:__align__|alignas)\(\d+\)", " ", line.split("__shared__", 1)[1])
        for part in re.sub(r"\[[^\]]*\]", "", body.rstrip(";")).split(","):
            out[re.findall(r"\w+", part)[-1]] = ok
    return out


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu*"))), ids=os.path.basename)
def test_wide_accesses_have_aligned_arrays(path):
    text = open(path).read()
    shared = _shared(text)
    names = {n for w in WIDE for n in w.findall(text)}
    assert [n for n in sorted(names) if shared.get(n) is False] == []
