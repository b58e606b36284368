"""Rules of the execution model that kernels keep and no run can show: they are
read from the sources."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "gpusteer_gb300" / "csrc"
SOURCES = sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh"))


def code(path):
    """The file without its comments."""
    text = re.sub(r"/\*.*?\*/", "", path.read_text(), flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def braced(text, at):
    """The balanced {...} block that opens at or after `at`."""
    start = text.index("{", at)
    depth = 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start:i + 1]
    raise ValueError("unbalanced braces")


def kernels(text):
    """(name, parameter list, body) of every __global__ function."""
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?"
                         r"(\w+)\s*\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), text[m.end():i - 1], braced(text, i)


def test_clusters_have_started_before_remote_shared_memory_is_touched():
    """A block may touch a peer's shared memory only after every block of the
    cluster runs, which a cluster barrier between the kernel's start and the
    first mapping of a peer's memory guarantees on every path that maps."""
    met = 0
    for path in SOURCES:
        for name, _, body in kernels(code(path)):
            for m in re.finditer(r"\bmap_shared_rank\b", body):
                met += 1
                # the code that every path to this mapping has passed: what
                # stands before it, without the closed blocks (their branches
                # need not have been taken)
                before, depth, kept = body[:m.start()], 0, []
                for c in reversed(before):
                    if c == "}":
                        depth += 1
                    elif c == "{":
                        depth -= depth > 0
                    elif depth == 0:
                        kept.append(c)
                passed = "".join(reversed(kept))
                assert re.search(r"\bcluster\.(sync|barrier_wait)\s*\(", passed), \
                    f"{path.name} {name}: {body[m.start() - 20:m.end() + 40]!r}"
    assert met >= 1


LAUNCHED_EARLY = sorted({m for p in SOURCES
                         for m in re.findall(r"\blaunch_after\(\s*(k_\w+)", code(p))} | {"k_db_cluster"})


def test_kernels_found():
    assert len(LAUNCHED_EARLY) >= 20
    assert any("*kern" in code(p) or "auto kern" in code(p) for p in SOURCES)  # named through a variable


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_no_read_only_path_loads(path):
    """A kernel whose blocks may be resident before its predecessor has ended
    reads what that predecessor writes: the read-only path is for data that
    nobody writes while the reading kernel runs."""
    text = code(path)
    for form in (r"__ldg\s*\(", r"ld\.global\.nc", r"__ldlu\s*\("):
        assert not re.search(form, text), f"{path.name}: {form}"


def test_early_launched_kernels_wait_first_and_take_no_invariant_pointers():
    """They begin with the wait, and no const __restrict__ pointer (whose
    loads count as invariant) is among their parameters or in the helpers that
    read the databases."""
    found = set()
    for path in SOURCES:
        text = code(path)
        for name, params, body in kernels(text):
            if name in LAUNCHED_EARLY or name == "k_fused":
                found.add(name)
                assert "__restrict__" not in params, f"{path.name} {name}"
                assert re.match(r"\{\s*after_previous\(\);", body), f"{path.name} {name}"
        if path.suffix == ".cuh" or path.name in ("gs_lists.cu", "gs_brute.cu", "gs_step.cu"):
            for m in re.finditer(r"__device__[^;{]*?\(([^;{]*?)\)\s*(?:const\s*)?\{", text):
                assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", m.group(1)), \
                    f"{path.name}: {m.group(0)[:120]}"
    assert found == set(LAUNCHED_EARLY) | {"k_fused"}


@pytest.mark.parametrize("path", SOURCES + sorted(CSRC.glob("*.h")), ids=lambda p: p.name)
def test_no_rule_holds_the_chips_sm_count(path):
    """Launch rules ask the device (sm_count)."""
    assert not re.search(r"\b152u?\b", code(path))
