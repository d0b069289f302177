"""Builds the CUDA library (libttt_b200.so) for sm_100a with nvcc, in-tree, and the native host path (_host.so).

    python -m ttt_rs_b200.build            # rebuild if any source is newer than the library
    python -m ttt_rs_b200.build --force
"""

from __future__ import annotations

import os
import re
import shutil
import subprocess
import sys
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "libttt_b200.so"
PROBE_SRC = CSRC / "probe_chain_latency.cu"      # stand-alone measurement program (bench.py --workload chain-latency)
PROBE_BIN = PKG / "build" / "probe_chain_latency"
SOURCES = ["ttt_abi.cu", "ttt_linear_fwd.cu", "ttt_linear_fwd_roles.cu", "ttt_linear_bwd.cu", "ttt_linear_bwd_f32.cu", "ttt_mlp_fwd.cu", "ttt_layer.cu", "ttt_layer_small.cu", "ttt_linear_partial.cu", "ttt_mlp_bwd.cu", "ttt_gemm.cu"]
HOST_SRC = CSRC / "ttt_host.cpp"                 # native host path of the Python operator, linked against LIB
HOST_LIB = PKG / "_host.so"
HOST_TAG = PKG / "build" / "_host.tag"           # what HOST_LIB was built against
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xptxas", "-v",
]
# Kernels whose groups of warps split the launch's registers among themselves (setmaxnreg): registers per thread that the
# splits add up to.  With fewer at launch a group would wait for registers that do not exist.
REGISTER_SPLITS = {"ttt_linear_bwd_f32.cu": ("ttt_linear_bwd_f32_kernel", 128)}


def check_register_split(src: str, log: str) -> None:
    """Raises unless every instantiation of `src`'s splitting kernel has exactly its registers in ptxas's report `log`."""
    if src not in REGISTER_SPLITS:
        return
    kernel, want = REGISTER_SPLITS[src]
    used = [int(n) for name, n in re.findall(r"Compiling entry function '(\w+)'.*?Used (\d+) registers", log, re.S) if kernel in name]
    if not used or any(n != want for n in used):
        raise RuntimeError(f"{src}: {kernel} must be built with {want} registers per thread, ptxas reports {used}")


def find_nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found (set NVCC or install the CUDA toolkit)")


def needs_build() -> bool:
    if not LIB.exists():
        return True
    t = LIB.stat().st_mtime
    deps = [p for p in CSRC.glob("*.cu") if p != PROBE_SRC] + list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h")) + \
        list((PKG.parent / "include").glob("*.h"))
    return any(p.stat().st_mtime > t for p in deps)


def build_probe(force: bool = False) -> Path:
    """The tensor-core chain-latency probe: its own executable, nothing of the library depends on it."""
    if not force and PROBE_BIN.exists() and PROBE_BIN.stat().st_mtime >= PROBE_SRC.stat().st_mtime:
        return PROBE_BIN
    PROBE_BIN.parent.mkdir(exist_ok=True)
    cmd = [find_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
           "-o", str(PROBE_BIN), str(PROBE_SRC)]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed on {PROBE_SRC.name}:\n{r.stdout}")
    return PROBE_BIN


def host_tag() -> str:
    """The interpreter and the torch that run this: `_host` uses the C++ interfaces of both, which change from one version
    to the next."""
    import sysconfig

    import torch
    return f"{sysconfig.get_config_var('EXT_SUFFIX')} torch {torch.__version__} {torch.version.git_version}\n"


def build_host(force: bool = False) -> Path:
    """The CPython extension module `_host`, for the interpreter and the torch that run this."""
    deps = [HOST_SRC, CSRC / "ttt_internal.h", PKG.parent / "include" / "ttt_b200.h"]
    tag = host_tag()
    if not force and HOST_LIB.exists() and all(HOST_LIB.stat().st_mtime >= p.stat().st_mtime for p in deps) \
            and HOST_TAG.exists() and HOST_TAG.read_text() == tag:
        return HOST_LIB
    import sysconfig

    import torch
    tdir = Path(torch.__file__).resolve().parent
    cuda = Path(find_nvcc()).resolve().parent.parent
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-Wno-attributes",
           f"-I{tdir}/include", f"-I{tdir}/include/torch/csrc/api/include", f"-I{cuda}/include",
           f"-I{sysconfig.get_paths()['include']}", str(HOST_SRC), "-o", str(HOST_LIB),
           f"-L{tdir}/lib", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda",
           f"-L{PKG}", f"-l:{LIB.name}", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed on {HOST_SRC.name}:\n{r.stdout}")
    HOST_TAG.parent.mkdir(exist_ok=True)
    HOST_TAG.write_text(tag)
    return HOST_LIB


def build(force: bool = False, verbose: bool = False) -> Path:
    build_probe(force)
    if not force and not needs_build():
        build_host(force)
        return LIB
    nvcc = find_nvcc()
    objs = []
    build_dir = PKG / "build"
    build_dir.mkdir(exist_ok=True)
    procs = []
    for src in SOURCES:
        obj = build_dir / (src + ".o")
        extra = os.environ.get("TTT_NVCC_EXTRA", "").split()
        cmd = [nvcc, *NVCC_FLAGS, *extra, "-c", str(CSRC / src), "-o", str(obj)]
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(str(obj))
    log = []
    for src, pr in procs:
        out, _ = pr.communicate()
        log.append(f"== {src}\n{out}")
        if pr.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{out}")
        check_register_split(src, out)
    cmd = [nvcc, "-shared", "-o", str(LIB), *objs]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}")
    build_host(force)
    (build_dir / "ptxas.log").write_text("\n".join(log))
    if verbose:
        print("\n".join(log))
    return LIB


if __name__ == "__main__":
    p = build(force="--force" in sys.argv, verbose=True)
    print(f"built {p}")
