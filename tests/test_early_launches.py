"""Early launches (launch_early, common.cuh): a kernel's blocks start before the previous kernel's
writes are complete, so each such kernel waits first, and no read of it, or of a device function
that it calls, may tell the compiler that the memory is constant while the kernel runs (const
__restrict__ parameters, __ldg, ld.global.nc): such a read could be moved above the wait. Read
from the sources, on the CPU."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "tsne-h2pack-python_b200" / "csrc"


def _close(s, i, pair):
    """Index behind the bracket that closes the one at s[i]."""
    depth = 0
    for j in range(i, len(s)):
        depth += (s[j] == pair[0]) - (s[j] == pair[1])
        if depth == 0:
            return j + 1
    raise AssertionError("unbalanced source")


def _functions():
    """name -> [(is kernel, parameters, body)] of the device code, and the names launched early."""
    found, early = {}, set()
    for f in sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh")):
        s = re.sub(r"//[^\n]*", "", f.read_text())
        s = re.sub(r"/\*.*?\*/", "", s, flags=re.S)
        early |= set(re.findall(r"\blaunch_early\(\s*(k_\w+)", s))
        for m in re.finditer(r"__(global|device)__\s[^;{}=]*?(?:__launch_bounds__\([^{;]*?\)\)?\s*)?\b(\w+)\s*\(", s):
            a = m.end() - 1
            if m.group(2) == "__launch_bounds__":    # the name is behind its bounds
                a = s.index("(", _close(s, a, "()"))
            name = re.search(r"(\w+)\s*$", s[:a]).group(1)
            b = _close(s, a, "()")
            tail = re.match(r"\s*(?:const)?\s*(?::[^{;]*)?\{", s[b:])
            if not tail:
                continue                             # a declaration
            o = b + tail.end() - 1
            found.setdefault(name, []).append((m.group(1) == "global", s[a:b], s[o + 1:_close(s, o, "{}") - 1]))
    return found, early


FUNCTIONS, EARLY = _functions()


def test_sources_are_read():
    assert {"k_attr_window", "k_bbox", "k_lists", "k_id2d", "k_id3", "k_down_leaves", "k_center"} <= EARLY
    assert all(any(k for k, _, _ in FUNCTIONS[n]) for n in EARLY), "every early kernel's definition is found"
    assert {"win_gather", "node_rec", "reduce_partials", "for_sources", "after_previous"} <= set(FUNCTIONS)


@pytest.mark.parametrize("name", sorted(EARLY))
def test_early_kernel_waits_first(name):
    for kernel, _, body in FUNCTIONS[name]:
        assert kernel and body.split(";")[0].strip() == "after_previous()"


@pytest.mark.parametrize("name", sorted(EARLY))
def test_early_kernel_reads_no_memory_as_constant(name):
    seen, todo = set(), [name]
    while todo:
        f = todo.pop()
        if f in seen:
            continue
        seen.add(f)
        for _, params, body in FUNCTIONS[f]:
            for bad in ("__restrict__", "__ldg", "global.nc"):
                assert bad not in params + body, f"{bad} in {f}, reached from {name}"
            todo += [c for c in set(re.findall(r"\b(\w+)\s*(?:<[\w\s,<>:]*>)?\s*\(", body)) if c in FUNCTIONS]


def test_every_thread_launches_early():
    """A served job takes the launch path that a direct run takes."""
    body = re.search(r"void launch_early\(.*?\n}\n", (CSRC / "common.cuh").read_text(), flags=re.S).group(0)
    assert "cfg.numAttrs = 1;" in body
    assert "thread_local" not in (CSRC / "common.cuh").read_text()
