"""Kernels that start under the end of the one in front: what they read is tied to their wait (``chain_wait`` in sm100_common.cuh)."""
import re

import pytest

from hetu_galvatron_b200.csrc import build

SM100 = build.CSRC / "sm100"


def overlapped_kernels(path):
    """(name, parameters, body) of every kernel of a file that calls ``chain_wait``."""
    for part in re.split(r"\b__global__\b", path.read_text())[1:]:
        head, body = part.split("{", 1)
        body = re.split(r"\n}\n", body, maxsplit=1)[0]
        head = re.sub(r"__launch_bounds__\([^()]*(\([^()]*\)[^()]*)*\)", "", head)
        if "chain_wait()" in body:
            name = re.search(r"(\w+)\s*\(", head)
            yield name.group(1), head[name.end():], body


# A `const ... __restrict__` pointer says that nothing writes behind it while the kernel runs, so that the compiler may read it
# before the wait; only an address that comes out of the wait rules that out.
@pytest.mark.parametrize("name", ["norm.cu", "elementwise.cu", "xent.cu"])
def test_restrict_inputs_are_tied_to_the_wait(name):
    kernels = list(overlapped_kernels(SM100 / name))
    assert kernels
    for kernel, params, body in kernels:
        inputs = re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", params)
        assert inputs, kernel
        loose = [p for p in inputs if not re.search(r"\b%s \+= [^;]*(zero|chain_wait\(\))" % p, body)]
        assert not loose, (kernel, loose)


# A load through the read-only path makes the same promise at the load itself.
@pytest.mark.parametrize("path", sorted([*SM100.glob("*.cu"), *SM100.glob("*.cuh")]), ids=lambda p: p.name)
def test_no_read_only_loads_behind_a_wait(path):
    text = re.sub(r"//.*", "", path.read_text())
    if path.suffix == ".cuh" or "chain_wait()" in text:
        assert not re.findall(r"__ldg\b|ld\.global\S*\.nc\b", text)
