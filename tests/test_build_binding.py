"""The torch marshalling module is rebuilt for another torch or Python, not only for newer sources."""
import importlib.util
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_binding_is_rebuilt_for_another_torch(tmp_path, monkeypatch):
    spec = importlib.util.spec_from_file_location("fmla_build", os.path.join(ROOT, "flashmla_windows_linux_sm120_b200", "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    binding = tmp_path / "_fmla_torch.so"
    binding.write_bytes(b"")
    monkeypatch.setattr(build, "BINDING_PATH", str(binding))
    monkeypatch.setattr(build, "OBJ_DIR", str(tmp_path))
    runs = []
    monkeypatch.setattr(build.subprocess, "run", lambda cmd, **kw: runs.append(cmd) or subprocess.CompletedProcess(cmd, 0, "", ""))
    build._build_binding(False)                     # newer than its sources, but for which torch is not known
    build._build_binding(False)
    assert len(runs) == 1
    stamp = tmp_path / "_fmla_torch.built_for"
    stamp.write_text(stamp.read_text().replace("__version__", "__other__"))
    build._build_binding(False)
    assert len(runs) == 2
