"""The in-tree build (csrc/build.py): what it needs, and what other processes see of it while it runs."""
from hetu_galvatron_b200.csrc import build


def test_host_modules_need_no_cuda_toolkit(monkeypatch, tmp_path):
    def missing():
        raise RuntimeError("nvcc not found")

    ran = []
    monkeypatch.setattr(build, "LIB_DIR", tmp_path)
    monkeypatch.setattr(build, "OBJ_DIR", tmp_path / "build")
    monkeypatch.setattr(build, "_nvcc", missing)
    monkeypatch.setattr(build, "_run", lambda cmd, log=None: ran.append(cmd))
    built = build.build_host()
    assert [p.name.split(".")[0] for p in built] == ["hg_dp_core", "hg_dataset_helpers"] and len(ran) == 2
