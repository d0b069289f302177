"""Kernels launched while the kernel before them on the stream drains: each waits for it (in the sources), and results do not
depend on what the host does between the launches (on the GPU)."""
import os
import re
import subprocess
import sys
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


def _kernels(text):
    for k in re.split(r"__global__\b", text)[1:]:
        name = re.search(r"\b(ttt_\w+_kernel)\(", k)
        if name:
            yield name.group(1), k


def test_a_kernel_that_does_not_wait_is_launched_behind_everything():
    """The backwards' scans let the reductions begin without having waited themselves: none of them may begin early, or two kernels
    behind one another would be unfinished when a third starts."""
    go, early = set(), set()
    for f in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//.*", "", f.read_text())
        go |= {n for n, k in _kernels(text) if "pdl_go()" in k and not re.search(r"\bpdl_(wait|join)\(\)", k)}
        for body in re.split(r"\n}\n", text):  # a function, or a kernel and its name
            if "__global__" in body:
                continue
            chosen = set(re.findall(r"kfn = [^;]*?\b(ttt_\w+_kernel)\b", body))
            for first in re.findall(r"launch_dependent\((.*?),", body):
                early |= chosen if first.strip() == "kfn" else set(re.findall(r"\bttt_\w+_kernel\b", first))
            if "ProgrammaticStreamSerialization" in body:
                early |= chosen
    assert go == {"ttt_linear_bwd_kernel", "ttt_linear_bwd_f32_kernel", "ttt_mlp_bwd_kernel"}
    assert {"ttt_gemm_bf16_tn_kernel", "ttt_layer_prologue_kernel", "ttt_linear_bwd_reduce_kernel", "ttt_linear_partial_kernel"} <= early
    assert not go & early


def test_a_kernel_that_waits_at_once_reads_nothing_before():
    header = (CSRC / "ttt_kernels.h").read_text()
    pointers = set(re.findall(r"\*\s*(\w+);", header))
    assert {"inner_out", "ln_w", "token_eta", "part_te"} <= pointers
    for f in sorted(CSRC.glob("*.cu")):
        for name, k in _kernels(re.sub(r"//.*", "", f.read_text())):
            if "pdl_join()" in k:
                for field in re.findall(r"\bp\.(\w+)\b(?!\s*[!=]= nullptr)", k[:k.index("pdl_join()")]):
                    assert field not in pointers, (name, field)


KINDS = ("linear bf16, streams alone", "linear bf16, streams sharing", "linear f32", "mlp", "layer 1x1001", "layer 13x56")


def _passes(kind, wait):
    """Eight passes on different inputs; `wait`: the host waits for each."""
    import ttt_rs_b200 as tb
    from oracle import ttt_oracle as O
    results = []
    for i in range(8):
        if kind.startswith("layer"):
            B, T = {"layer 1x1001": (1, 1001), "layer 13x56": (13, 56)}[kind]
            if i == 0:
                torch.manual_seed(7)
                cfg = tb.TTTLayerConfig(hidden_size=768, num_heads=12)
                layer = tb.TTT(cfg, device="cuda", dtype=torch.bfloat16)
                inner = tb.new_inner(cfg, device="cuda", dtype=torch.bfloat16, allow_partial=True)
            x = (torch.randn(B, T, 768, generator=torch.Generator().manual_seed(i)) * 0.5).to("cuda", torch.bfloat16)
            with torch.no_grad():
                results.append([layer(x, inner, inner.init_state(B))])
        elif kind == "mlp":
            t = {k: v.cuda() for k, v in O.make_inputs(2, 4, 48, 64, 16, seed=i, dtype=torch.bfloat16, inner="mlp").items()}
            cfg = tb.FusedTttConfig.new(16, 64, 1e-6, 256, 1)
            a = (t["xq"], t["xk"], t["xv"], tb.TTTMLPState(t["w1"], t["b1"], t["w2"], t["b2"]), t["token_eta"], t["ttt_lr_eta"],
                 t["ln_weight"], t["ln_bias"])
            ws = tb.mlp_backward_workspace(t["xq"], cfg)
            out, _ = tb.fused_ttt_mlp_forward(*a, cfg, backward_workspace=ws)
            g = tb.fused_ttt_mlp_backward(*a, t["grad_output"], cfg, workspace_from_forward=ws)
            results.append([out] + [g[k] for k in sorted(g) if k.startswith("grad_")])
        else:
            B, dtype = {"linear bf16, streams alone": (2, torch.bfloat16), "linear bf16, streams sharing": (16, torch.bfloat16),
                        "linear f32": (2, torch.float32)}[kind]
            t = {k: v.cuda() for k, v in O.make_inputs(B, 12, 64, 64, 16, seed=i, dtype=dtype).items()}
            cfg = tb.FusedTttConfig.new(16, 64, 1e-6, 64, 2)
            names = ("xq", "xk", "xv", "weight", "bias", "token_eta", "ttt_lr_eta", "ln_weight", "ln_bias")
            ins = tb.TttInputs(*[t[k] for k in names])
            outs, saved = tb.TttTileMultiKernel.forward_launch(ins, cfg)
            grads = tb.TttTileMultiKernel.backward_launch(saved, tb.TttOutputs(t["grad_output"], None, None), cfg)
            results.append([outs.output, *[getattr(grads, k) for k in names]])
        if wait:
            torch.cuda.synchronize()
    torch.cuda.synchronize()
    tb.TttTileMultiKernel.check_status()
    return [[x.cpu() for x in r] for r in results]


@pytest.mark.gpu
def test_passes_back_to_back_equal_launches_one_at_a_time(tmp_path):
    """Training passes of the three backwards, whose reductions begin while the scans drain, and layer calls: enqueued without a pause,
    against a process in which every launch has ended before the next one is made (CUDA_LAUNCH_BLOCKING)."""
    want = tmp_path / "one_at_a_time.pt"
    code = (f"import sys, torch; sys.path[:0] = [{str(Path(__file__).resolve().parent)!r}, {str(CSRC.parent.parent)!r}]; "
            f"import test_dependent_launches as t; torch.save({{k: t._passes(k, True) for k in t.KINDS}}, {str(want)!r})")
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300, env={**os.environ, "CUDA_LAUNCH_BLOCKING": "1"})
    one_at_a_time = torch.load(want)
    for kind in KINDS:
        for i, (a, b) in enumerate(zip(one_at_a_time[kind], _passes(kind, False))):
            assert len(a) == len(b) and all(torch.equal(x, y) for x, y in zip(a, b)), (kind, i)
