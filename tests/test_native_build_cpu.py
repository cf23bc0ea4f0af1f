"""The in-tree build (csrc/build.py): what it needs, and what other processes see of it while it runs."""
import re
import threading
import time
import zlib
from pathlib import Path

import pytest
import torch

from hetu_galvatron_b200.csrc import build


@pytest.fixture
def tree(monkeypatch, tmp_path):
    """An empty tree, and the commands that were run for it: each writes to its output twice."""
    ran = []

    def run(cmd, log=None):
        ran.append(cmd)
        out = Path(cmd[cmd.index("-o") + 1])
        out.write_text("half")
        time.sleep(0.2)
        assert not list(tmp_path.glob("hg_*.so")) or len(ran) > 1        # nothing to be seen of the first one yet
        out.write_text("whole")

    monkeypatch.setattr(build, "LIB_DIR", tmp_path)
    monkeypatch.setattr(build, "OBJ_DIR", tmp_path / "build")
    monkeypatch.setattr(build, "_run", run)
    return tmp_path, ran


def test_host_modules_need_no_cuda_toolkit(tree, monkeypatch):
    def missing():
        raise RuntimeError("nvcc not found")

    monkeypatch.setattr(build, "_nvcc", missing)
    built = build.build_host()
    assert [p.name.split(".")[0] for p in built] == ["hg_dp_core", "hg_dataset_helpers"] and len(tree[1]) == 2


def test_outputs_appear_whole_and_once(tree):
    first, second = (threading.Thread(target=build.build_host) for _ in range(2))
    first.start(), second.start()
    first.join(), second.join()
    files = sorted(p.name.split(".")[0] for p in tree[0].iterdir() if p.is_file())
    assert files == ["hg_dataset_helpers", "hg_dp_core"] and len(tree[1]) == 2
    assert all(p.read_text() == "whole" for p in tree[0].iterdir() if p.is_file())


def test_a_failed_compiler_leaves_nothing(tree, monkeypatch):
    def fails(cmd, log=None):
        Path(cmd[cmd.index("-o") + 1]).write_text("half")
        raise RuntimeError("command failed")

    monkeypatch.setattr(build, "_run", fails)
    with pytest.raises(RuntimeError):
        build.build_host()
    assert not [p for p in tree[0].iterdir() if p.is_file()]


def test_a_built_tree_that_cannot_be_written_to(tree, monkeypatch):
    build.build_host()
    monkeypatch.setattr(build, "OBJ_DIR", tree[0] / "nowhere" / "build")
    assert len(build.build_host()) == 2 and len(tree[1]) == 2


def test_autograd_nodes_of_another_build_are_built_again(tree, monkeypatch):
    torch_ops = build.build_torch_ops()
    version = int(re.search(r"kHgNativeInterface = (\d+)", (build.CSRC / "sm100" / "native_interface.h").read_text()).group(1))
    assert build.torch_ops_current(version) and not build.torch_ops_current(version + 1)
    build.build_torch_ops()
    assert len(tree[1]) == 1
    monkeypatch.setattr(torch, "__version__", torch.__version__ + "x")                 # another torch
    assert not build.torch_ops_current(version)
    build.build_torch_ops()
    assert len(tree[1]) == 2 and build.torch_ops_current(version)
    torch_ops.rename(torch_ops.with_name("hg_torch_ops.cpython-00-elsewhere.so"))      # another interpreter
    assert not build.torch_ops_current(version, unmarked=True)


# Raise kHgNativeInterface with any change that turns up here, and note the new sum beside it.
INTERFACES = {1: 633082835, 2: 3060780885, 3: 945623936, 4: 3301874251, 5: 2171609436, 6: 2350616146, 7: 1669815742}


def test_entry_points_that_the_nodes_call_by_address():
    """Their argument lists are those of the library, and a change of them is a new version of the interface."""
    def kinds(params):
        return "".join("p" if "*" in p or re.match(r"\s*[VA]\b", p) else {"int": "i", "long long": "l", "float": "f"}[
            re.match(r"\s*(int|long long|float)\b", p).group(1)] for p in params.split(","))

    nodes = (build.CSRC / "host" / "torch_ops.cpp").read_text()
    kernels = "".join(p.read_text() for p in sorted((build.CSRC / "sm100").glob("*.cu")))
    slots = dict(re.findall(r"\(\*(\w+)\)\(([^)]*)\);", nodes.split("struct Kernels {")[1].split("};")[0]))
    called = []
    for name, slot in re.findall(r'at\("(hg_\w+)", K\.(\w+)\)', nodes):
        params = re.search(r"\b%s\(([^)]*)\)\s*\{" % name, kernels).group(1)
        assert kinds(params) == kinds(slots[slot]), name
        called.append(name + ":" + kinds(params))
    assert len(called) == len(slots)
    structs = [re.sub(r"//.*|\s+", " ", (build.CSRC / "sm100" / h).read_text()) for h in ("attn_tensor.h", "decoder_step.h")]
    version = int(re.search(r"kHgNativeInterface = (\d+)", (build.CSRC / "sm100" / "native_interface.h").read_text()).group(1))
    assert INTERFACES[version] == zlib.crc32(" ".join(sorted(called) + structs).encode())
