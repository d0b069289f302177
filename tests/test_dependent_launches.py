"""Kernels launched while the kernel before them on the stream drains: each waits for it (in the sources), and results do not
depend on what the host does between the launches (on the GPU)."""
import re
from pathlib import Path

import pytest
import torch

CSRC = Path(__file__).resolve().parent.parent / "ttt_rs_b200" / "csrc"


def test_every_kernel_that_may_begin_early_waits():
    waiting, launched = {}, set()
    for f in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//.*", "", f.read_text())
        for k in re.split(r"__global__\b", text)[1:]:
            name = re.search(r"\b(ttt_\w+_kernel)\(", k)
            if name and re.search(r"\bpdl_(wait|join)\(\)", k):
                waiting[name.group(1)] = k
        if "launch_dependent(" in text or "ProgrammaticStreamSerialization" in text:
            launched |= {m for m in re.findall(r"launch_dependent\((?:[^;]*?)\b(ttt_\w+_kernel)\b", text)}
            if "launch_dependent(kfn" in text:  # (instantiations picked into `kfn` beforehand)
                launched |= set(re.findall(r"kfn = [^;]*?\b(ttt_\w+_kernel)\b", text)) - {"ttt_layer_epilogue_bwd_kernel"}
    assert launched <= set(waiting), launched - set(waiting)
    joined = {n for n, k in waiting.items() if "pdl_join()" in k}
    assert joined == {"ttt_gemm_bf16_tn_kernel", "ttt_layer_prologue_kernel", "ttt_layer_epilogue_kernel", "ttt_linear_fwd_roles_kernel",
                      "ttt_linear_bwd_reduce_kernel", "ttt_mlp_bwd_reduce_kernel"}
    for n in joined:  # what the kernel before may still write is never read as read-only data
        assert not re.search(r"\b(?:ldg4|__ldg)\(|ld\.global\.nc", waiting[n]), n


@pytest.mark.gpu
@pytest.mark.parametrize("B,H,T,gate", [(1, 12, 1001, False), (3, 16, 43, True), (40, 12, 1, True), (13, 12, 56, False)])
def test_layer_calls_back_to_back_equal_calls_one_by_one(B, H, T, gate):
    """A prompt of ragged length, a short one, a token per sequence and more streams than SMs with a remainder: sixteen calls on
    different inputs enqueued without a pause, temporaries of one reused by the next, against the same calls each waited for."""
    import ttt_rs_b200 as tb
    torch.manual_seed(B * T)
    cfg = tb.TTTLayerConfig(hidden_size=H * 64, num_heads=H, use_gate=gate)
    layer = tb.TTT(cfg, device="cuda", dtype=torch.bfloat16)
    inner = tb.new_inner(cfg, device="cuda", dtype=torch.bfloat16, allow_partial=True)
    xs = [torch.randn(B, T, H * 64, device="cuda", dtype=torch.bfloat16) * 0.5 for _ in range(16)]
    with torch.no_grad():
        one_by_one = []
        for x in xs:
            one_by_one.append(layer(x, inner, inner.init_state(B)))
            torch.cuda.synchronize()
        queued = [layer(x, inner, inner.init_state(B)) for x in xs]
        torch.cuda.synchronize()
    tb.TttTileMultiKernel.check_status()
    for a, b in zip(one_by_one, queued):
        assert torch.equal(a, b)
