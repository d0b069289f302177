"""The native host path is rebuilt when the torch or the interpreter it was built against has changed."""
import subprocess

from ttt_rs_b200 import build as B


def test_a_changed_torch_or_interpreter_rebuilds_the_host_path(monkeypatch, tmp_path):
    import torch
    lib = tmp_path / "_host.so"
    monkeypatch.setattr(B, "HOST_LIB", lib)
    monkeypatch.setattr(B, "HOST_TAG", tmp_path / "build" / "_host.tag", raising=False)
    runs = []

    def compiler(cmd, **kw):
        runs.append(cmd)
        lib.write_bytes(b"")
        return subprocess.CompletedProcess(cmd, 0, "")

    monkeypatch.setattr(B.subprocess, "run", compiler)
    B.build_host()
    B.build_host()
    assert len(runs) == 1
    monkeypatch.setattr(torch, "__version__", "99.0")
    B.build_host()
    B.build_host()
    assert len(runs) == 2
