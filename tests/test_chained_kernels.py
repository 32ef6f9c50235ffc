"""The rules of chain.h in the sources: a kernel that is launched before its predecessor's writes are flushed waits
in its first statement and reads nothing through a pointer declared free of aliases, not even in the functions
that are inlined into it."""
import pathlib
import re

import pytest

SRC = pathlib.Path(__file__).resolve().parent.parent / "ugacc_gb300" / "csrc"


def _code(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


def _kernels():
    """(name, parameters, body) of every __global__ function."""
    for path in sorted(SRC.glob("*.cu")):
        text = _code(path)
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)+\s*)?(\w+)\(", text):
            depth, k = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[k], 0)
                k += 1
            params, start = text[m.end():k], text.index("{", k)
            depth, e = 1, start + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[e], 0)
                e += 1
            yield m.group(1), params, text[start + 1:e - 1]


KERNELS = {name: (params, body) for name, params, body in _kernels()}
LAUNCHED = sorted({m for path in SRC.glob("*.cu") for m in re.findall(r"launch_chained\(\s*(\w+)", _code(path))}
                  - {"void"})


def test_kernels_are_found():
    assert len(LAUNCHED) > 20 and set(LAUNCHED) <= set(KERNELS)


@pytest.mark.parametrize("name", LAUNCHED)
def test_chained_kernel(name):
    params, body = KERNELS[name]
    # shared-memory declarations may stand before the wait: they access nothing
    first = re.sub(r"^(\s*(extern\s+)?__shared__[^;]*;)*\s*", "", body)
    assert first.startswith("chain_enter();"), first[:60]
    assert "__restrict__" not in params + body


@pytest.mark.parametrize("header", ["pairs.h", "dgemm_tile.h", "chain.h"])
def test_functions_inlined_into_chained_kernels(header):
    assert "__restrict__" not in _code(SRC / header)
