"""Kernels follow each other by programmatic dependent launch: that is only sound when every kernel waits for the one before it
in every thread, ahead of any early return, and when no launch goes round the helper that asks for it."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "dgen-audio_b200", "csrc")


def _bodies(text):
    """What follows the opening brace of every kernel definition."""
    for m in re.finditer(r"__global__", text):
        i, depth = m.end(), 0
        while depth or text[i] not in "{;":
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        if text[i] == "{":
            yield text[m.start():i].strip(), text[i + 1:].lstrip()


def test_every_kernel_waits_for_the_one_before_it_first_thing():
    seen = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        if os.path.basename(path) == "blocks.cu":      # writes the source of generated blocks, which are launched plainly
            continue
        with open(path) as f:
            text = f.read()
        assert "<<<" not in text, path
        for head, body in _bodies(text):
            assert body.startswith("dgc_after_previous();"), (path, head)
            seen += 1
    assert seen > 90
