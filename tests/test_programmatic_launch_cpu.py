"""Kernels that may start while their predecessor drains (programmatic dependent launch), checked in their sources.

What such a kernel reads may be written by the kernel before it until ``pdl_wait()`` returns, so no statement above that
call may reach through a pointer, and no thread may leave before it: a kernel that completed early would let the kernel
after it start before the kernel before it is done.
"""

import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "nano_omni_b200" / "csrc"


def _closing(text, at, pair):
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise AssertionError("unbalanced source")


def kernels(path):
    """(name, parameter list, body) of every __global__ function, comments removed."""
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)
    for match in re.finditer(r"__global__", text):
        launch_bounds = re.match(r"(?:\s*(?:void|__\w+__\s*\([^()]*(?:\([^()]*\)[^()]*)*\)))*\s*", text[match.end() :])
        at = match.end() + launch_bounds.end()
        name = re.match(r"\w+", text[at:]).group()
        end = _closing(text, text.index("(", at), "()")
        begin = text.index("{", end)
        yield name, text[at + len(name) + 1 : end], text[begin + 1 : _closing(text, begin, "{}")]


WAITING = [
    (path.name, name, parameters, body)
    for path in sorted(CSRC.glob("*.cu"))
    for name, parameters, body in kernels(path)
    if "pdl_wait()" in body
]


def test_kernels_are_found():
    names = {name for _, name, _, _ in WAITING}
    assert {"fa_fwd_bf16_kernel", "fa_fwd_i8f8_kernel", "matmul_kernel", "quantize_qk_kernel", "sol_select_kernel"} <= names


@pytest.mark.parametrize("file,name,parameters,body", WAITING, ids=[f"{f}:{n}" for f, n, _, _ in WAITING])
def test_nothing_is_read_before_the_wait(file, name, parameters, body):
    before = body[: body.index("pdl_wait()")]
    for parameter in parameters.split(","):
        word = re.search(r"(\w+)\s*$", parameter).group(1)
        if "*" in parameter:
            assert not re.search(rf"\b{word}\b", before), f"{name} touches {word} before the wait"
        else:  # a record of sizes and pointers: its members may be copied, not reached through
            assert not re.search(rf"\b{word}\.\w+\s*(\[|->)|[=(,;{{]\s*\*\s*{word}\.\w+", before), f"{name} reads through {word}"
        # loads that the compiler may take for constant could be moved above the wait
        assert not ("const" in parameter and "__restrict__" in parameter), f"{name}: {word}"
    assert "__ldg" not in body
    assert not re.search(r"\breturn\b", before), "a thread may leave before the wait"


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu")), ids=lambda p: p.name)
def test_dependent_launches_name_kernels_that_wait(path):
    text = path.read_text()
    waiting = {name for file, name, _, _ in WAITING if file == path.name}
    launches = [m.group(1) for m in re.finditer(r"launch_pdl\(\s*[^,]+,\s*([^,;]+)", text)]
    for target in launches:
        names = {n for n, _, _ in kernels(path) if re.search(rf"\b{n}\b", target)}
        if not names:  # through a local variable: every kernel that may be assigned to it
            assigned = re.findall(rf"\b{target.strip()}\s*=([^;]*);", text)
            names = {n for n, _, _ in kernels(path) if any(re.search(rf"\b{n}\b", a) for a in assigned)}
        assert names and names <= waiting, f"{path.name}: {target.strip()} is launched as a dependent without a wait"
