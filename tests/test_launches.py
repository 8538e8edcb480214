"""Kernels launched with programmatic stream serialisation have to begin with
pdl_wait(): without it they would start beside the kernel before them."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "icls-release_b200" / "csrc"
TEXT = {f.name: re.sub(r"//[^\n]*", "", f.read_text()) for f in sorted(CSRC.iterdir()) if f.suffix in (".cu", ".cuh")}


def closing(s, i, pair="()"):
    """index of the bracket that closes the one at i"""
    depth = 0
    for k in range(i, len(s)):
        depth += (s[k] == pair[0]) - (s[k] == pair[1])
        if not depth:
            return k
    raise ValueError(s[i:i + 80])


def kernels(s):
    """(name, body) of every kernel defined in s"""
    for m in re.finditer(r"__global__\s+void\s+", s):
        i = m.end()
        if s.startswith("__launch_bounds__", i):
            i = closing(s, s.index("(", i)) + 1
        p = s.index("(", i)
        body = s[closing(s, p) + 1:].lstrip()
        if body.startswith("{"):
            yield s[i:p].strip(), body[1:].lstrip()


@pytest.mark.parametrize("name", [n for n, s in TEXT.items() if "pdl(" in s])
def test_overlapped_kernels_wait_first(name):
    s = TEXT[name]
    launched = set(re.findall(r"\bpdl\((k_\w+)", s))
    if re.search(r"\bpdl\(kernel\b", s):  # through a generic lambda: any of the file's
        launched |= {k for k, _ in kernels(s)}
    waits = {k: body.startswith("pdl_wait();") for t in TEXT.values() for k, body in kernels(t)}
    if name != "icls_common.cuh":
        assert launched
    for k in launched:
        assert waits[k], k


@pytest.mark.parametrize("name", list(TEXT))
def test_device_memory_is_set_on_the_streams_that_use_it(name):
    """The contexts' and networks' streams do not wait for the legacy stream,
    and a memset or a copy from pageable memory there may still be under way
    when it returns: no memset goes there, and no copy to the device but the
    constants', which are waited for."""
    s = TEXT[name]
    assert not re.search(r"\bcudaMemset\(", s)
    assert not re.search(r"\bcudaMemcpy\([^;]*cudaMemcpyHostToDevice", s)
    for m in re.finditer(r"\bcudaMemcpyToSymbol\(", s):
        assert "cudaStreamSynchronize(nullptr)" in s[m.end():m.end() + 400]
