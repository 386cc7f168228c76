"""What the CUDA sources must not contain, since nothing at run time would show it."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCES = sorted(glob.glob(os.path.join(ROOT, "wtb_gb300", "csrc", "*.cu*")))
FUNCTION = re.compile(r"^(?:template[^\n]*\n)?__(?:global|device)__[^;{]*?\b(\w+)\(([^{};]*)\)\s*\{(.*?)^\}", re.M | re.S)


def functions(path):
    """name -> (parameters, body) of the file's kernels and device functions"""
    with open(path) as f:
        text = re.sub(r"//[^\n]*|__(launch_bounds|cluster_dims)__\((\([^()]*\)|[^()])*\)", "", f.read())
    return {m.group(1): (m.group(2), m.group(3)) for m in FUNCTION.finditer(text)}


def test_early_started_kernels_take_no_restrict_pointers():
    """A kernel that starts before its predecessor has ended reads what that one still writes: a restrict pointer would let
    the compiler move such a load above the wait, or take it from the read-only path."""
    early = 0
    for path in SOURCES:
        fns = functions(path)
        waits = {n for n, (_, b) in fns.items() if "griddepcontrol.wait" in b or "cudaGridDependencySynchronize" in b}
        for name, (params, body) in fns.items():
            if not any(re.search(r"\b%s\(" % w, body) for w in waits):
                continue
            early += 1
            assert "__restrict__" not in params, name
            for callee, (callee_params, _) in fns.items():
                if re.search(r"\b%s\(" % callee, body):
                    assert "__restrict__" not in callee_params, (name, callee)
    assert early >= 2  # the dense reduction's two kernels a column


def test_shuffle_masks_are_not_taken_from_the_active_lanes():
    """Which lanes are active after a loop of different trip counts is the compiler's choice: a mask names its lanes."""
    for path in SOURCES:
        with open(path) as f:
            assert "__activemask" not in f.read(), path
