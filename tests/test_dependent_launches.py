"""What a launch that may begin before the one before it is complete asks of
its kernel, read from the sources: the wait comes first, no parameter promises
that memory stays as it is during the kernel (const with __restrict__), nothing
is read through the non-coherent path, and a kernel without the wait is
launched plainly.
"""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "fluids3_gb300" / "csrc"


def matching(text: str, at: int, pair: str = "()") -> int:
    depth = 0
    for k in range(at, len(text)):
        depth += (text[k] == pair[0]) - (text[k] == pair[1])
        if depth == 0:
            return k
    raise AssertionError("unbalanced")


def code(path: Path) -> str:
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)


def kernels():
    for path in sorted(CSRC.glob("*.cu")):
        text = code(path)
        for m in re.finditer(r"__global__", text):
            head = re.compile(r"\b(k_\w+)\s*\(").search(text, m.start())
            end = matching(text, head.end() - 1)
            body = text[end + 1:].lstrip()
            assert body.startswith("{")
            yield path.name, head.group(1), text[head.end():end], body[1:].lstrip()


KERNELS = list(kernels())


def test_the_sources_hold_kernels_of_both_kinds():
    waits = {name for _, name, _, body in KERNELS if body.startswith("follow_previous();")}
    assert {"k_density", "k_force_advance", "k_scan", "k_adj_force"} <= waits
    assert {"k_sample_bricks", "k_density_pairs"} & waits == set()


@pytest.mark.parametrize("file,name,params,body", KERNELS, ids=[f"{f}:{n}" for f, n, _, _ in KERNELS])
def test_a_kernel_that_waits_promises_nothing_about_memory_before_it(file, name, params, body):
    if "follow_previous()" not in body[: matching("{" + body, 0, "{}")]:
        return
    assert body.startswith("follow_previous();"), "the wait is not the first statement"
    assert "__restrict__" not in params


def test_nothing_is_read_through_the_non_coherent_path():
    for path in sorted(list(CSRC.glob("*.cu")) + list(CSRC.glob("*.cuh"))):
        assert not re.search(r"ld\.global\.nc|__ldg\s*\(", code(path)), path.name


def test_kernels_without_the_wait_are_launched_plainly():
    plain = [(f, n) for f, n, _, body in KERNELS if not body.startswith("follow_previous();")]
    assert plain
    for file, name in plain:
        text = code(CSRC / file)
        naming = []
        for m in re.finditer(r"\b" + name + r"\b", text):
            # the function that names it, to its end
            function = text[text.rfind("\n}", 0, m.start()) + 1:text.find("\n}", m.start())]
            if "__global__" not in function:
                naming.append(function)
                assert not re.search(r"(?<!int )\blaunch\s*\(", function), f"{file}: {name}"
        assert any("<<<" in f for f in naming), f"{file}: {name}"
