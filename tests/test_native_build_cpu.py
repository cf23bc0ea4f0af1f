"""The in-tree build (csrc/build.py): what it needs, and what other processes see of it while it runs."""
import threading
import time
from pathlib import Path

import pytest

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
