"""In-tree build of the C-ABI library: nvcc, sm_100a only.

``python flashmla_windows_linux_sm120_b200/build.py`` (run as a script, so that a stale library cannot block its own rebuild) compiles
``csrc/*.cu`` into ``flashmla_windows_linux_sm120_b200/lib/libflashmla_b200.so`` and the torch marshalling module
``csrc/torch_binding.cpp`` into ``lib/_fmla_torch.so``, which finds the library beside it.
Objects are rebuilt only when a source or header is newer, the module also when torch or Python is another one.
"""
from __future__ import annotations

import concurrent.futures
import glob
import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
LIB_DIR = os.path.join(PKG_DIR, "lib")
OBJ_DIR = os.path.join(PKG_DIR, "build")
LIB_PATH = os.path.join(LIB_DIR, "libflashmla_b200.so")
BINDING_PATH = os.path.join(LIB_DIR, "_fmla_torch.so")
INCLUDE_DIR = os.path.join(os.path.dirname(PKG_DIR), "include")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "--use_fast_math",
    "-std=c++17", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found; the library must be built where the CUDA toolkit is installed")
    return cand


def _newest(paths) -> float:
    return max(os.path.getmtime(p) for p in paths)


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(LIB_DIR, exist_ok=True)
    os.makedirs(OBJ_DIR, exist_ok=True)
    sources = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    headers = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h")) + \
        glob.glob(os.path.join(INCLUDE_DIR, "*.h"))
    hdr_time = _newest(headers) if headers else 0.0
    nvcc = _nvcc()
    jobs = []
    for src in sources:
        obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")
        stale = force or not os.path.exists(obj) or os.path.getmtime(obj) < max(os.path.getmtime(src), hdr_time)
        if stale:
            jobs.append((src, obj))

    def compile_one(job):
        src, obj = job
        extra = os.environ.get("FMLA_EXTRA_NVCC_FLAGS", "").split()     # e.g. -DFMLA_TRACE for a timeline build
        cmd = [nvcc] + NVCC_FLAGS + extra + ["-I", INCLUDE_DIR, "-c", src, "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
        return r.stderr

    if jobs:
        with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
            for out in ex.map(compile_one, jobs):
                if verbose and out:
                    print(out, file=sys.stderr)
    objs = [os.path.join(OBJ_DIR, os.path.basename(s)[:-3] + ".o") for s in sources]
    if jobs or not os.path.exists(LIB_PATH) or os.path.getmtime(LIB_PATH) < _newest(objs):
        cmd = [nvcc, "-shared", "-o", LIB_PATH] + objs + ["-gencode", "arch=compute_100a,code=sm_100a", "-lcudart"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    _build_binding(force)
    return LIB_PATH


def _build_binding(force: bool) -> None:
    src = os.path.join(CSRC, "torch_binding.cpp")
    header = os.path.join(INCLUDE_DIR, "flashmla_b200.h")
    # torch is located, not imported: importing it takes longer than this compilation
    torch_dir = os.path.dirname(importlib.util.find_spec("torch").origin)
    # the module holds on to the ABI of one torch and one Python
    with open(os.path.join(torch_dir, "version.py")) as f:
        built_for = f"{sys.version}\n{torch_dir}\n{f.read()}"
    stamp = os.path.join(OBJ_DIR, "_fmla_torch.built_for")
    if not force and os.path.exists(BINDING_PATH) and os.path.getmtime(BINDING_PATH) >= _newest([src, header]) and os.path.exists(stamp):
        with open(stamp) as f:
            if f.read() == built_for:
                return
    cuda_home = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", src, "-o", BINDING_PATH,
           "-I", sysconfig.get_paths()["include"], "-I", os.path.join(torch_dir, "include"),
           "-I", os.path.join(torch_dir, "include", "torch", "csrc", "api", "include"),
           "-I", os.path.join(cuda_home, "include"),
           "-L", os.path.join(torch_dir, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python",
           "-L", LIB_DIR, "-l:libflashmla_b200.so", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"building {BINDING_PATH} failed:\n{r.stdout}\n{r.stderr}")
    with open(stamp, "w") as f:
        f.write(built_for)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
