"""Warp votes, shuffles and matches of the kernels name the lanes that take part.

A mask from __activemask() holds the lanes that happened to run together when
it was read.  Nothing keeps them together until the next instruction, so a vote
over it from divergent code may name lanes that never reach it, which is
undefined and may wait for ever.  Running such a kernel shows nothing (it
works until it hangs), so this reads the sources."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qsl_gb300", "csrc")
SYNC = re.compile(r"__(?:all|any|ballot|shfl(?:_up|_down|_xor)?|match_any|match_all|reduce_\w+)_sync\(([^,()]*(?:\([^()]*\))?)")


def test_no_mask_comes_from_activemask():
    masks = []
    for name in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, name)) as f:
            code = re.sub(r"//[^\n]*", "", f.read())
        assert "__activemask" not in code and "activemask.b32" not in code, name
        masks += [(name, m.group(1).strip().lower()) for m in SYNC.finditer(code)]
    assert masks
    assert {m for _, m in masks} == {"0xffffffffu"}, masks
