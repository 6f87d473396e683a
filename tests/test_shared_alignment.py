"""Shared arrays that the CUDA sources read or write in pieces wider than their element say how they are aligned: without it the place that the
compiler happens to give them decides whether such an access faults."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nano-vllm-rs_b200", "csrc")
SIZE = {"float": 4, "int": 4, "unsigned": 4, "int32_t": 4, "uint32_t": 4, "bf16": 2, "uint8_t": 1, "unsigned char": 1, "double": 8, "int64_t": 8, "uint64_t": 8,
        "unsigned long long": 8, "float2": 8, "uint2": 8, "float4": 16, "uint4": 16, "int4": 16, "bf162": 4}


def wide_accesses(text):
    """(array, bytes it is aligned to, bytes of the widest access) of every static shared array that is accessed through a cast."""
    out = []
    for align, kind, names in re.findall(r"__shared__\s+(?:__align__\((\d+)\)\s+)?((?:unsigned )?(?:long long|\w+))\s+([^;]+);", text):
        if kind not in SIZE:
            continue
        for name in re.findall(r"(\w+)\s*\[", re.sub(r"\[[^\]]*\]", "[", names)):
            casts = re.findall(r"reinterpret_cast<\s*(?:const\s+)?(?:volatile\s+)?(\w+)\s*\*>\(\s*&?%s\b" % name, text)
            widest = max([SIZE.get(c, 0) for c in casts], default=0)
            if widest:
                out.append((name, max(int(align or 0), SIZE[kind]), widest))
    return out


def test_shared_arrays_are_aligned_for_their_widest_access():
    found = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "**", "*.cu*"), recursive=True)):
        text = re.sub(r"extern __shared__[^;]*;", "", re.sub(r"//[^\n]*", "", open(path).read()))
        for name, have, need in wide_accesses(text):
            found += 1
            assert have >= need, f"{os.path.basename(path)}: {name} is aligned to {have} bytes and accessed in {need}"
    assert found > 0
