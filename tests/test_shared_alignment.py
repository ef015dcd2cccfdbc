"""Shared arrays that a kernel reads or writes in vectors are declared with the vector's alignment: without it an array lies where the
others leave it, and a change to one of those can misalign it (CPU, from the sources)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ittai_b200", "csrc")
SIZE = {"bf16": 2, "float": 4, "int": 4, "uint32_t": 4, "int32_t": 4, "float2": 8, "uint2": 8, "float4": 16, "uint4": 16, "int4": 16, "unsigned long long": 8}
ARRAY = re.compile(r"__shared__\s+(?:__align__\((\d+)\)\s+)?(?:volatile\s+)?(unsigned long long|\w+)\s+([^;]*);")
VECTOR = re.compile(r"reinterpret_cast<(?:const\s+)?(float2|float4|uint2|uint4|int4|uint32_t)\s*\*>\(\s*&?(\w+)")


def _misaligned(text):
    """``(array, alignment, needed)`` for every shared array that is accessed in wider pieces than its declaration allows."""
    text = re.sub(r"//[^\n]*", "", text)
    bad = []
    for kernel in re.split(r"\n(?=template|__global__)", text):          # names are a kernel's own
        arrays = {}
        for align, kind, names in ARRAY.findall(kernel):
            for name in re.findall(r"(\w+)\s*(?=\[)", names):
                arrays[name] = int(align) if align else SIZE.get(kind, 1)
        for vector, name in VECTOR.findall(kernel):
            if name in arrays and arrays[name] < SIZE[vector]:
                bad.append((name, arrays[name], SIZE[vector]))
    return bad


@pytest.mark.parametrize("source", sorted(os.path.basename(p) for p in glob.glob(os.path.join(CSRC, "*.cu*"))))
def test_vectors_are_aligned(source):
    with open(os.path.join(CSRC, source)) as f:
        assert not _misaligned(f.read())
