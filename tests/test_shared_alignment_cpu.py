"""A kernel that reads its dynamic shared memory in 16-byte pieces declares it on 16 bytes: without that the array starts where the
static one ends, and the first __shared__ variable that someone adds makes the loads misaligned."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "dgen-audio_b200", "csrc")
NARROW = re.compile(r"extern __shared__ (?!__align__\((?:16|32|64|128)\))(float|char|uint8_t) (\w+)\[\]")


def _kernels(text):
    for m in re.finditer(r"__global__", text):
        i, depth = m.end(), 0
        while depth or text[i] not in "{;":
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        if text[i] == ";":
            continue
        start = i
        while True:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
            if depth == 0:
                break
        yield text[m.start():start], text[start:i]


def test_wide_reads_of_dynamic_shared_memory_are_declared_on_their_size():
    seen = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        with open(path) as f:
            text = f.read()
        for head, body in _kernels(text):
            if "extern __shared__" not in body:
                continue
            seen += 1
            # float4 views of shared memory only: global pointers are loaded through __ldg, __ldcs or a named global row
            wide = re.search(r"reinterpret_cast<(?:const )?(?:float4|uint4|int4) \*>\((?:sm|sh|xc|st|stage|gs)\b", body)
            assert not (wide and NARROW.search(body)), (os.path.basename(path), " ".join(head.split())[:120])
    assert seen >= 15
