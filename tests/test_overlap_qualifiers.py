"""Kernels that are launched to overlap with the launch before them (htcuda.cu launch(true, ...)) may not
promise the compiler that what that launch writes is read-only: a `const ... __restrict__` pointer may be
read through the non-coherent path, which needs data that is constant from the kernel's first block on.
Only what the caller wrote before the call's first launch may carry the promise. CPU only."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hypertrace_b200", "csrc", "htcuda.cu")
WRITTEN_BEFORE_THE_CALL = {"scene", "views", "order"}


def _text():
    with open(SRC) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _balanced(text, at):
    """The text inside the parentheses that open at `at`."""
    depth = 0
    for i in range(at, len(text)):
        depth += {"(": 1, ")": -1}.get(text[i], 0)
        if depth == 0:
            return text[at + 1:i]
    raise AssertionError("unbalanced")


def test_overlapped_kernels_promise_nothing_about_their_predecessors_output():
    text = _text()
    kernels = {}
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__(?=\())?", text):
        at = m.end()
        if text[at] == "(":
            at += len(_balanced(text, at)) + 2
        name = re.match(r"\s*(\w+)\s*", text[at:])
        kernels[name.group(1)] = _balanced(text, at + name.end())
    overlapped = set()
    for m in re.finditer(r"\blaunch\(true,", text):
        call = _balanced(text, m.start() + len("launch"))
        overlapped |= set(re.findall(r"\w+", call)) & set(kernels)
    assert {"render_wave", "render_batch_wave", "k_sort_scatter", "k_bsort_scatter"} <= overlapped
    for name in overlapped:
        for param in kernels[name].split(","):
            if "const" in param.split("*")[0] and "__restrict__" in param:
                assert re.findall(r"\w+", param)[-1] in WRITTEN_BEFORE_THE_CALL, (name, param.strip())
