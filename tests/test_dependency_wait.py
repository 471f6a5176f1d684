"""Every kernel of the library starts while its predecessors still run and waits for them on the device
(griddepcontrol.wait).  What it reads afterwards was written during its own lifetime, so no load may be declared read-only:
a `const __restrict__` parameter, `__ldg` or `ld.global.nc` lets the compiler move it above the wait, where it sees the call
before.  These checks read the sources."""
import re

import pytest

from conftest import ROOT

CSRC = ROOT / "fused_moe_b200" / "csrc"
SOURCES = sorted(p for p in CSRC.iterdir() if p.suffix in (".cu", ".cuh"))


def code_of(path):
    text = re.sub(r"/\*.*?\*/", "", path.read_text(), flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def kernels_of(code):
    """(name, parameters, body) of each __global__ function."""
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^;{]*?\)\s*)?(\w+)\s*\(", code):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(code[i], 0)
            i += 1
        params = code[m.end():i - 1]
        start = code.index("{", i)
        depth, j = 1, start + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(code[j], 0)
            j += 1
        yield m.group(1), params, code[start:j]


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_no_load_is_declared_read_only(path):
    code = code_of(path)
    found = [w for w in ("__restrict__", "__ldg", "__ldca", "__ldcg", "ld.global.nc") if w in code]
    assert not found


def test_every_kernel_waits():
    found = {}
    for path in SOURCES:
        for name, _, body in kernels_of(code_of(path)):
            found[name] = "pdl_wait()" in body
    assert len(found) >= 16
    assert all(found.values()), [n for n, ok in found.items() if not ok]


def test_pointer_parameters_are_read_through_the_ordered_loads():
    """A const pointer parameter is used as an argument of ld_dep / ld_l2 / ld_stream / route_token / copy_row / the
    half-row reader, in an address computation or a null test, never dereferenced by itself."""
    for path in SOURCES:
        for name, params, body in kernels_of(code_of(path)):
            for p in re.findall(r"const\s+\w+\s*\*\s*(\w+)", params):
                assert not re.search(rf"(?<![\w.&]){p}\s*\[", body), (name, p)
                assert not re.search(rf"[=(,!]\s*\*\s*{p}\b", body), (name, p)
                for m in re.finditer(rf"(?<![\w.]){p}\s*->", body):
                    assert body[:m.start()].endswith("ld_l2(&"), (name, p)
