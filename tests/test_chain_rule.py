"""Kernels that start before their predecessor's memory is visible (chain.cuh):
read from the sources, no GPU."""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "leopard_em_gb300", "csrc")


def _chained_kernels():
    """(file, name, parameters, body) of every kernel that calls chain_wait()."""
    out = []
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, f)) as src:
            text = re.sub(r"//[^\n]*", "", src.read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", text):
            params = text[m.end() : text.index(")", m.end())]
            body = _block(text[text.index("{", m.end()) :])
            if "chain_wait()" in body:
                out.append((f, m[1], params, body))
    return out


def _block(text):
    """The braced block that text starts with."""
    depth = 0
    for i, ch in enumerate(text):
        depth += (ch == "{") - (ch == "}")
        if depth == 0:
            return text[: i + 1]
    raise AssertionError("unbalanced braces")


def _without_lambdas(text):
    """What runs where it stands: lambdas read the pointers where they are called."""
    while m := re.search(r"auto \w+ = \[&\]\([^)]*\) *(?=\{)", text):
        text = text[: m.start()] + text[m.end() + len(_block(text[m.end() :])) :]
    return text


def test_every_kernel_launched_as_a_link_waits():
    """A link without the wait would let the one after it run ahead of everything before."""
    waiting = {name for _, name, _, _ in _chained_kernels()}
    launched = set()
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")) and f != "chain.cuh":
            with open(os.path.join(CSRC, f)) as src:
                text = src.read()
            for m in re.finditer(r"launch_chained\(\s*(\w+)", text):
                # a variable holds one of the kernels named where it is set
                names = {m[1]} if m[1].endswith("_kernel") else set(
                    re.findall(r"\w+_kernel", re.search(rf"auto\*? {m[1]} = ([^;]*);", text)[1]))
                assert names
                launched |= names
    assert len(launched) >= 15 and launched <= waiting


@pytest.mark.parametrize("kernel", _chained_kernels(), ids=lambda k: k[1])
def test_restrict_pointers_are_passed_on_after_the_wait(kernel):
    """A __restrict__ pointer that the wait has not seen may be read (or written)
    above it: each has to go through LGB_CHAIN_POINTER after the wait, and
    nothing may be read through it before."""
    _, _, params, body = kernel
    names = [re.search(r"(\w+)\s*$", p)[1] for p in params.split(",") if "__restrict__" in p]
    before, after = body.split("chain_wait()", 1)
    before = _without_lambdas(before)
    assert "return" not in before  # every thread waits
    for n in names:
        assert f"LGB_CHAIN_POINTER({n})" in after, n
        for use in re.finditer(rf"\b{n}\b", before):  # (whether it is null may be asked)
            assert before[: use.start()].endswith("if ("), f"{n} is used before the wait"
