"""Kernels that wait for their predecessor on the device (pdl_wait) may start
while it still writes, so what they read has to be loaded by ordinary loads: a
non-coherent load (__ldg, or one the compiler derives from a const restrict
pointer) promises data that is constant from the kernel's start to its end, and
such a load need not stay behind the wait. Checked on the sources: no function
that such a kernel reaches may use either."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "aerodynamics4mc-fabric_b200" / "csrc"


def source(path: Path) -> str:
    text = re.sub(r"/\*.*?\*/", " ", path.read_text(), flags=re.S)
    text = re.sub(r"//[^\n]*", " ", text)
    return re.sub(r'(?<!include )"[^"\n]*"', '""', text)


def with_includes(path: Path, seen: dict[Path, str]) -> dict[Path, str]:
    if path not in seen and path.exists():
        seen[path] = source(path)
        for name in re.findall(r'#include "([^"]+)"', seen[path]):
            with_includes((path.parent / name).resolve(), seen)
    return seen


def matching(text: str, at: int, pair: str) -> int:
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise ValueError("unbalanced")


def functions(text: str) -> list[tuple[str, str, str]]:
    """(name, parameters, body) of every function defined in the text."""
    out = []
    for m in re.finditer(r"\b([A-Za-z_]\w*)\s*\(", text):
        if m.group(1) in ("if", "for", "while", "switch", "return", "sizeof", "__launch_bounds__", "__maxnreg__"):
            continue
        close = matching(text, m.end() - 1, "()")
        body = re.match(r"\s*(?:const\s*)?(?::[^{;]*)?\{", text[close + 1:])
        if body:
            start = close + 1 + body.end() - 1
            out.append((m.group(1), text[m.end():close], text[start:matching(text, start, "{}") + 1]))
    return out


def waiting_kernels_reach(unit: str) -> dict[str, list[tuple[str, str]]]:
    """Per kernel of the unit that waits: the (name, text) of all functions it reaches by name."""
    defs: dict[str, list[str]] = {}
    for text in with_includes(CSRC / unit, {}).values():
        for name, params, body in functions(text):
            defs.setdefault(name, []).append(params + " " + body)
    reach = {}
    for kernel, texts in defs.items():
        if kernel in ("pdl_wait", "launch_pdl") or not any("pdl_wait()" in t for t in texts):
            continue
        todo, seen = [kernel], set()
        while todo:
            name = todo.pop()
            if name in seen:
                continue
            seen.add(name)
            for t in defs[name]:
                todo += [c for c in set(re.findall(r"\b([A-Za-z_]\w*)\b", t)) if c in defs]
        reach[kernel] = [(name, t) for name in sorted(seen) for t in defs[name]]
    return reach


@pytest.mark.parametrize("unit,kernels", [
    ("meso_exact.cu", {"meso_collide_kernel", "meso_ambient_kernel", "meso_stream_kernel"}),
    ("d3q27_exact.cu", {"step_ip2_kernel"}),
    ("d3q27_fast.cu", {"step_ip2_kernel"}),
    ("thermal_exact.cu", {"thermal_update_kernel", "thermal_fill_kernel"}),
    ("batch.cu", {"batch_step_kernel"}),
])
def test_waiting_kernels_use_ordinary_loads(unit, kernels):
    reach = waiting_kernels_reach(unit)
    assert kernels <= set(reach)
    bad = sorted({f"{kernel}: {name}" for kernel, parts in reach.items() for name, t in parts
                  if "__ldg" in t or re.search(r"const\s+[\w:<>\s]*\*\s*__restrict__", t)})
    assert not bad, bad
