"""What the kernels of programmatic dependent launches have to keep to, read from their source (no GPU)."""
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


SOURCES = sorted(p for p in CSRC.rglob("*.cu") if "wait_for_producers" in p.read_text())
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
