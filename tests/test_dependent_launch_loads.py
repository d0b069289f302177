"""Kernels launched with programmatic dependent launch begin while the kernel before them still writes their input: only
weights may go through the non-coherent load path there (its data must not be written while the kernel runs)."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "ttt_rs_b200" / "csrc"
SETTLED = {"ttt_layer_small_out_kernel": ("w +", "static_cast<const __nv_bfloat16*>(p.ln_w)", "static_cast<const __nv_bfloat16*>(p.ln_b)")}


def test_only_settled_weights_take_the_non_coherent_path():
    seen = 0
    for f in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//.*", "", f.read_text())
        kernels = re.split(r"__global__\b", text)[1:]
        for k in kernels:
            if "pdl_wait()" not in k:
                continue
            seen += 1
            name = re.search(r"\b(ttt_\w+_kernel)\(", k).group(1)
            for arg in re.findall(r"\b(?:ldg4|__ldg)\(([^;]*)", k):
                assert arg.startswith(SETTLED.get(name, ())), f"{f.name}: {name} reads {arg[:60]!r} as read-only data"
    assert seen == 3  # projections, inner step, output
