"""Kernels launched ahead of the end of the kernel before them (csrc/pdl.cuh) may
read nothing through a pointer that the compiler is free to read before the
wait.  A __restrict__ parameter allows that, so each is made opaque by the wait
itself: every kernel that waits names all of its __restrict__ pointers there."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "cuda-lbm-ibm-fvm_b200" / "csrc"
# null in the instance that carries the attribute
UNUSED = {("k_predict2", "kap")}


def kernels(text):
    """(name, parameter list, body) of the __global__ functions."""
    text = re.sub(r"//[^\n]*", "", text)

    def closing(i, a, b):
        depth = 0
        for j in range(i, len(text)):
            depth += (text[j] == a) - (text[j] == b)
            if depth == 0:
                return j
        raise ValueError(text[i:i + 80])

    for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(", text):
        end = closing(m.end() - 1, "(", ")")
        brace = text.index("{", end)
        yield m.group(1), text[m.end():end], text[brace:closing(brace, "{", "}")]


@pytest.mark.parametrize("source", sorted(p.name for p in CSRC.glob("*.cu") if "pdl_enter" in p.read_text()))
def test_restrict_pointers_are_opaque_after_the_wait(source):
    found = 0
    for name, params, body in kernels((CSRC / source).read_text()):
        wait = re.search(r"pdl_enter\(([^)]*)\)", body)
        if not wait:
            continue
        found += 1
        named = {a.strip() for a in wait.group(1).split(",")}
        pointers = {re.search(r"(\w+)\s*$", p).group(1) for p in params.split(",") if "__restrict__" in p}
        missing = {p for p in pointers - named if (name, p) not in UNUSED}
        assert not missing, (name, sorted(missing))
    assert found
