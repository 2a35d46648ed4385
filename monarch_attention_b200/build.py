"""Build the C-ABI shared library (sm_100a only) in-tree with nvcc, and the Python binding on top of it.

    python -m monarch_attention_b200.build [--force] [--verbose]

Output: monarch_attention_b200/lib/libmonarch_attention_b200.so and monarch_attention_b200/_native.so
"""
from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB_DIR = os.path.join(PKG, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libmonarch_attention_b200.so")
NATIVE_PATH = os.path.join(PKG, "_native.so")
NATIVE_SOURCE = "ma_torch.cpp"
SOURCES = ["ma_api.cu", "ma_generic.cu", "ma_tc.cu", "ma_fused.cu", "ma_warp.cu", "ma_warp_f32.cu", "ma_head.cu", "ma_head_f16.cu", "ma_head_states.cu", "ma_head_states_f16.cu", "ma_tile.cu", "ma_flow.cu", "ma_flow_f16.cu", "ma_backward.cu", "ma_backward_f16.cu", "ma_backward_f32.cu", "ma_noalloc.cu", "ma_host.cu"]
HEADERS = ["ma_common.cuh", "ma_tile_common.cuh", "ma_flow.inc", "ma_head.inc", "ma_backward.inc", "ma_warp_common.cuh", "ma_warp_kernels.inc", "ma_warp_head.inc", "ma_warp_wide.inc", "ma_sm100.cuh", "ma_tc_plan.cuh", os.path.join("..", "..", "include", "monarch_attention_b200.h")]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
    "--expt-relaxed-constexpr",
]


def find_nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found (set NVCC=/path/to/nvcc)")


def _newest(names) -> float:
    return max(os.path.getmtime(os.path.join(CSRC, n)) for n in names)


def _older(path: str, than: float) -> bool:
    return not os.path.exists(path) or os.path.getmtime(path) < than


def _native_command(obj: str) -> list[str]:
    from torch.utils.cpp_extension import include_paths
    inc = [f"-I{p}" for p in include_paths() + ["/usr/local/cuda/include", sysconfig.get_paths()["include"]]]
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-DTORCH_API_INCLUDE_EXTENSION_H",
            "-DTORCH_EXTENSION_NAME=_native", *inc, "-c", os.path.join(CSRC, NATIVE_SOURCE), "-o", obj]


def build(force: bool = False, verbose: bool = False) -> str:
    """Compiles what is older than its sources: the headers count for every source."""
    os.makedirs(LIB_DIR, exist_ok=True)
    common = max(_newest(HEADERS), os.path.getmtime(os.path.abspath(__file__)))
    jobs, objs = [], []
    for src in [NATIVE_SOURCE] + SOURCES:
        obj = os.path.join(LIB_DIR, os.path.splitext(src)[0] + ".o")
        if src != NATIVE_SOURCE:
            objs.append(obj)
        if not force and not _older(obj, max(common, _newest([src]))):
            continue
        if src == NATIVE_SOURCE:
            cmd = _native_command(obj)
        else:
            cmd = [find_nvcc(), *(["-Xptxas", "-v"] if verbose else []), *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
        jobs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in jobs:
        out, _ = p.communicate()
        if p.returncode != 0 or verbose:
            print(f"--- {src} ---\n{out}", file=sys.stderr)
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("compilation failed")
    newest = max(os.path.getmtime(o) for o in objs)
    if _older(LIB_PATH, newest):
        subprocess.check_call([find_nvcc(), "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC",
                               "-o", LIB_PATH, *objs, "-cudart", "static"])
    native_obj = os.path.join(LIB_DIR, os.path.splitext(NATIVE_SOURCE)[0] + ".o")
    if _older(NATIVE_PATH, os.path.getmtime(native_obj)):
        from torch.utils.cpp_extension import library_paths
        subprocess.check_call(["g++", "-shared", "-o", NATIVE_PATH, native_obj, f"-L{LIB_DIR}", "-l:" + os.path.basename(LIB_PATH),
                               "-Wl,-rpath,$ORIGIN/lib", *(f"-L{p}" for p in library_paths()), "-lc10", "-lc10_cuda",
                               "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python"])
    return LIB_PATH


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(force=a.force, verbose=a.verbose))
