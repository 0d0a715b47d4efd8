"""Order of the steps on which the tiled kernels' tensor memory depends, read from
their source: a wrong order shows only as a rare hang or a stale value on the
GPU."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "provekit_b200",
                    "csrc")


def code(name):
    """A source file without its comments."""
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)


def body(text, function):
    """The body of the first definition of function in text."""
    at = text.index("{", re.search(r"\b%s\([^;{]*\)[^;{]*\{" % function, text).start())
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[at + 1:i]
    raise AssertionError(f"{function}: unbalanced braces")


def test_no_columns_are_held_while_waiting_for_a_kernel():
    """A CTA that waits for the previous kernel holds no tensor memory that this
    kernel may still need, and a dependent kernel starts only when every CTA
    has its own: wait, allocate, barrier, trigger."""
    text = code("tc_reduce.cuh")
    steps = body(text, "open")
    for part in ("begin", "ready"):
        if re.search(r"\b%s\(sh[^)]*\);" % part, steps):
            steps = re.sub(r"\b%s\(sh[^)]*\);" % part, lambda m: body(text, part), steps)
    order = [steps.index(s) for s in ("griddepcontrol.wait", "tcgen05.alloc", "__syncthreads()",
                                      "griddepcontrol.launch_dependents")]
    assert order == sorted(order)


def test_columns_are_allocated_and_kernels_triggered_in_one_place():
    all_code = "".join(code(os.path.basename(f)) for f in glob.glob(os.path.join(CSRC, "*.cu*")))
    for step in ("tcgen05.alloc.", "griddepcontrol.launch_dependents", "griddepcontrol.wait"):
        assert all_code.count(step) == 1, step


def calls(text):
    """Names of the calls in text by where they end: arguments come before the call."""
    found = []
    for m in re.finditer(r"\b(\w+)\s*(?:<\w+>)?\s*\(", text):
        depth, at = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[at], 0)
            at += 1
        found.append((at, m.group(1)))
    return [name for _, name in sorted(found)]


def accesses(text, function):
    """Tensor memory's stores, waits for them and loads in the order of the source,
    calls of the text's own functions followed."""
    names = set(re.findall(r"\b(\w+)\s*\([^;{}()]*\)\s*(?:const\s*)?\{", text))
    out = []
    for name in calls(body(text, function)):
        if name.startswith("tmem_st"):
            out.append("store")
        elif name == "tmem_written":
            out.append("wait")
        elif name.startswith("tmem_ld"):
            out.append("load")
        elif name in names - {"if", "for", "while", function}:
            out += accesses(text, name)
    return out


@pytest.mark.parametrize("source,function", [("poseidon2.cu", "permute"),
                                             ("sky_tc.cuh", "compress"), ("sky_tc.cuh", "permute")])
def test_stores_are_complete_before_the_next_load(source, function):
    """tcgen05.st is asynchronous: a tcgen05.ld after it without tcgen05.wait::st in
    between may read what was there before."""
    order = accesses(code(source) + code("tc_reduce.cuh"), function)
    assert {"store", "wait", "load"} <= set(order)
    pending = False
    for step in order:
        assert not (step == "load" and pending)
        pending = step == "store" or (pending and step != "wait")
