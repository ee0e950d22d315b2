"""Words that blocks wait on: in CUDA's memory model an acquiring load pairs
with releases of the same word only if both access the same bytes, so a word
is polled at the width it is released at. Read from the kernels' source.
"""

import os
import re

import fastlbp_b200

CSRC = os.path.join(os.path.dirname(os.path.abspath(fastlbp_b200.__file__)), "csrc")


def test_polls_and_releases_have_one_width():
    seen = 0
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, f)) as fh:
            text = fh.read()
        polled = set(re.findall(r"ld\.acquire\.gpu\.global\.[bu](\d+)", text))
        released = set(re.findall(r"(?:red|atom|st)\.release\.gpu\.global(?:\.\w+)?\.[bu](\d+)", text))
        seen += len(polled)
        assert polled == released, (f, polled, released)
    assert seen
