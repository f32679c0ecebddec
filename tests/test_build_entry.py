"""build() compiles the reference's substep only from a tree that holds it."""
import importlib.util
import os

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_a_tree_without_the_reference(monkeypatch, tmp_path):
    spec = importlib.util.spec_from_file_location("graft_entry", os.path.join(ROOT, "__graft_entry__.py"))
    entry = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(entry)
    from mpm_cuda_b200 import build
    calls = []
    monkeypatch.setattr(build, "build", lambda force: None)
    monkeypatch.setattr(entry.subprocess, "run", lambda cmd, check: calls.append(cmd))
    monkeypatch.setenv("MPM_REFERENCE_TREE", str(tmp_path))
    entry.build()
    assert len(calls) == 1 and "liboracle.so" in calls[0]
    (tmp_path / "src" / "simulator").mkdir(parents=True)
    (tmp_path / "src" / "simulator" / "MPMCUDA.cu").write_text("")
    entry.build()
    assert len(calls) == 3 and calls[2][-1] == f"REF={tmp_path}"
