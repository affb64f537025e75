"""CUDA guarantees that another CTA's shared memory exists only once that CTA is known to run: every kernel of the
library that maps it has to pass a cluster barrier before its first access.  Which access comes first in time is read
from the source: helpers (lambdas) count where they are called, everything else where it stands."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "xped_gb300" / "csrc"
BARRIER = re.compile(r"\b(?:cl|cluster)\.(?:sync|barrier_wait)\(\)")
LAMBDA = re.compile(r"auto (\w+) = \[&\]\([^)]*\)(?: mutable)? \{")


def block(text, at):
    """The braces that open at or after `at`, as (start, end)."""
    a = text.index("{", at)
    depth = 0
    for i in range(a, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return a, i
    raise AssertionError("unbalanced braces")


def functions():
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"^(?:__global__|__device__)[^;{}]*\)\s*\{", text, re.M | re.S):
            a, b = block(text, m.end() - 1)
            if "map_shared_rank" in text[a:b]:
                name = re.sub(r"__launch_bounds__\([^)]*\)", "", m.group(0)).split("(")[0].split()[-1]
                yield pytest.param(text[a:b], id=f"{path.name}:{name}")


@pytest.mark.parametrize("body", list(functions()))
def test_a_cluster_barrier_comes_before_the_first_access_to_another_cta(body):
    helpers = {}
    for m in LAMBDA.finditer(body):
        a, b = block(body, m.end() - 1)
        helpers[m.group(1)] = (a, b)
    accesses = []
    for m in re.finditer(r"map_shared_rank", body):
        inside = [n for n, (a, b) in helpers.items() if a < m.start() < b]
        if not inside:
            accesses.append(m.start())
        for n in inside:
            accesses += [c.start() for c in re.finditer(rf"\b{n}\(", body) if not helpers[n][0] < c.start() < helpers[n][1]]
    first = BARRIER.search(body)
    assert first is not None and first.start() < min(accesses)


def test_the_kernels_are_found():
    assert len(list(functions())) >= 4
