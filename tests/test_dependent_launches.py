"""What the kernels of programmatic dependent launches have to keep to, read from their source (no GPU).

Such a kernel may run while the kernel in front of it still writes.  A load through a `const T *__restrict__` parameter, or
through __ldg, counts as one of memory that nobody writes during the kernel, so a compiler may move it in front of the wait:
wait_for_producers() has to be given every such parameter, and no kernel behind a wait loads non-coherently."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "evo.cpp_b200" / "csrc"
FUNCTION = re.compile(r"(__global__|__device__)\s+(?:__forceinline__\s+)?(?:void|bool|int|float|auto|[\w:]+(?:<[^<>]*>)?)\s+"
                      r"(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(")


def _matching(text: str, at: int, pair: str) -> int:
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise AssertionError("unbalanced source")


def _functions(path: Path):
    """{name: (is a kernel, parameters, body)} of the device functions of a file."""
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)
    found = {}
    for match in FUNCTION.finditer(text):
        end = _matching(text, match.end() - 1, "()")
        begin = re.compile(r"[\s{;]").match(text, end + 1) and text.find("{", end)
        if text[end + 1:begin].strip() not in ("", "const"):
            continue  # a declaration
        found[match[2]] = (match[1] == "__global__", text[match.end():end], text[begin:_matching(text, begin, "{}") + 1])
    return found


def _reached(functions, name, seen=None):
    seen = set() if seen is None else seen
    seen.add(name)
    for other in functions:
        if other not in seen and re.search(rf"\b{other}\b", functions[name][2]):
            _reached(functions, other, seen)
    return seen


SOURCES = sorted(p for p in CSRC.rglob("*.cu") if "wait_for_producers" in p.read_text())


def test_the_instructions_have_one_home():
    users = [p.name for p in CSRC.rglob("*.cu*") if "griddepcontrol" in p.read_text()]
    assert users == ["common.cuh"]
    assert len(SOURCES) >= 10


READ_AND_WRITTEN = {"cache", "state"}  # of the parameters that are not const


def _named(body: str) -> set:
    return set(re.findall(r"\w+", " ".join(re.findall(r"wait_for_producers\(([^)]*)\)", body))))


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_outputs_stay_apart_from_what_is_read(path):
    """What a kernel only writes depends on what it has read, so it needs no order of its own; made opaque, it could be
    the memory of every load behind it, and those would wait for its stores."""
    for name, (kernel, parameters, body) in _functions(path).items():
        if kernel:
            written = set(re.findall(r"__restrict__\s*(\w+)", re.sub(r"const [\w:]+ \*__restrict__\s*\w+", "", parameters)))
            assert not (written - READ_AND_WRITTEN) & _named(body), name


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_waiting_kernels_load_behind_their_wait(path):
    functions = _functions(path)
    waiting = [n for n, (kernel, _, body) in functions.items() if kernel and "wait_for_producers" in body]
    assert waiting
    for name in waiting:
        _, parameters, body = functions[name]
        named = _named(body)
        read = set(re.findall(r"const [\w:]+ \*__restrict__\s*(\w+)", parameters))
        read |= READ_AND_WRITTEN & set(re.findall(r"__restrict__\s*(\w+)", parameters))
        assert read <= named, (name, read - named)
        for function in _reached(functions, name):
            assert not re.search(r"__ldg\b|ld\.global\.nc", functions[function][2]), (name, function)


@pytest.mark.parametrize("path", SOURCES + [CSRC / "qgmma_emulation.cu"], ids=lambda p: p.name)
def test_kernels_that_release_without_a_wait_are_launched_plainly(path):
    """Their completion would say nothing about the kernels further back."""
    functions = _functions(path)
    silent = [n for n, (kernel, _, body) in functions.items()
              if kernel and "release_dependents" in body and "wait_for_producers" not in body]
    if silent:
        assert "launch_dependent(" not in path.read_text(), silent
