"""Compile the CUDA library in-tree for sm_100a (nvcc cross-compiles without a GPU)."""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libtyr_b200_attn.so")
CALLS_PATH = os.path.join(LIB_DIR, "_calls.so")   # the Python call layer: a CPython extension over the C ABI
CALLS_SOURCE = "py_calls.cpp"
SOURCES = ["api.cu", "prefill_sm100.cu", "backward_sm100.cu", "decode_splitkv.cu", "check_fp32.cu", "qk_prologue.cu",
           "stalled_wait.cu"]
HEADERS = ["ptx_sm100.cuh", "mma_sync.cuh", "attn_internal.h", "scan_plan.h", "unit_parts.h",
           os.path.join("..", "..", "include", "tyr_b200_attn.h")]

# The reference's own nvcc flags for GPU=B200 (cc/Makefile:66-76) minus fast-math
# (the kernels ask for approximate ex2/lg2 explicitly where they want them) and
# minus the ThunderKittens define.
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-std=c++17", "-O3", "--expt-relaxed-constexpr", "-lineinfo",
    "-Xcompiler", "-fPIC", "-shared",
]


def nvcc_path() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found: the attention library cannot be built")
    return nvcc


def _older(path: str, deps) -> bool:
    if not os.path.exists(path):
        return True
    t = os.path.getmtime(path)
    return any(os.path.getmtime(os.path.join(CSRC, d)) > t for d in deps)


def library_stale() -> bool:
    return _older(LIB_PATH, SOURCES + HEADERS)


def _calls_command():
    """g++ command of the call layer.  It sees the C ABI's header only and is linked against the library next to it.
    None where it cannot be built: the C ABI needs neither g++ nor a torch with CUDA, the Python calls need both."""
    try:
        import torch
    except ImportError:
        return None
    if torch.version.cuda is None or shutil.which("g++") is None:
        return None
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(nvcc_path()))
    return (["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
             f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
             f"-I{root}/include", f"-I{root}/include/torch/csrc/api/include", f"-I{cuda}/include",
             "-I" + sysconfig.get_paths()["include"], os.path.join(CSRC, CALLS_SOURCE), "-o", CALLS_PATH,
             f"-L{LIB_DIR}", "-l:" + os.path.basename(LIB_PATH), f"-L{root}/lib", "-ltorch_python", "-ltorch", "-ltorch_cpu",
             "-ltorch_cuda", "-lc10", "-lc10_cuda", "-Wl,-rpath,$ORIGIN"])


def _calls_stamp() -> str:
    """What the call layer's binary interface depends on beside its sources."""
    import torch
    return f"python {sys.version}\ntorch {torch.__version__} {torch.version.git_version}\n"


def calls_stale() -> bool:
    """The call layer is missing, older than its sources, or built for another Python or torch (and can be built)."""
    if _calls_command() is None:
        return False
    if _older(CALLS_PATH, [CALLS_SOURCE, HEADERS[-1]]) or not os.path.exists(CALLS_PATH + ".built_for"):
        return True
    with open(CALLS_PATH + ".built_for") as f:
        return f.read() != _calls_stamp()


def stale() -> bool:
    return library_stale() or calls_stale()


def build(force: bool = False, verbose: bool = False) -> str:
    """Build lib/libtyr_b200_attn.so, and the Python call layer where it can be built, if missing or stale."""
    os.makedirs(LIB_DIR, exist_ok=True)

    def run(cmd):
        res = subprocess.run(cmd, capture_output=True, text=True)
        if verbose:
            print(res.stderr)
        if res.returncode != 0:
            raise RuntimeError(os.path.basename(cmd[0]) + " failed:\n" + res.stderr)

    if force or library_stale():
        run([nvcc_path()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) +
            ["-o", LIB_PATH] + [os.path.join(CSRC, f) for f in SOURCES])
    if force or calls_stale():
        cmd = _calls_command()
        if cmd is not None:
            run(cmd)
            with open(CALLS_PATH + ".built_for", "w") as f:
                f.write(_calls_stamp())
    return LIB_PATH


if __name__ == "__main__":
    print(build(force=True, verbose=True))
