"""The native host path is rebuilt when the torch or the interpreter it was built against has changed; a kernel that splits
its registers among groups of warps is only built with the count that the split needs."""
import subprocess

import pytest

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


@pytest.mark.parametrize("counts,ok", (((128, 128), True), ((128, 120), False), ((168,), False), ((), False)))
def test_a_register_split_needs_its_count(counts, ok):
    src, kernel = "ttt_linear_bwd_f32.cu", "ttt_linear_bwd_f32_kernel"
    # (as ptxas -v reports them, another kernel of the file in front)
    log = "ptxas info    : Compiling entry function '_Z5otherv' for 'sm_100a'\nptxas info    : Used 40 registers\n" + "".join(
        f"ptxas info    : Compiling entry function '_ZN3ttt25{kernel}ILi{i}E' for 'sm_100a'\n"
        f"ptxas info    : Function properties for x\n    0 bytes stack frame\nptxas info    : Used {n} registers, used 5 barriers\n"
        for i, n in enumerate(counts))
    if ok:
        B.check_register_split(src, log)
        B.check_register_split("ttt_gemm.cu", "")  # (a file without such a kernel)
    else:
        with pytest.raises(RuntimeError):
            B.check_register_split(src, log)
