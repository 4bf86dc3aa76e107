"""Build the two native parts in-tree, into landmark_attention_b200/lib/:

  libb200lmk.so   the kernels behind a plain C ABI (nvcc for sm_100a, no torch involved).  Each source is compiled to an
                  object file (in parallel, only when it or a header changed) and the objects are linked.
  _lmk_host.so    the host layer on PyTorch's C++ API (g++): checks, allocations, autograd nodes.  It looks the C ABI up in
                  libb200lmk.so at run time.
"""
import os
import shutil
import subprocess
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
OBJ_DIR = os.path.join(HERE, "_obj")
LIB_PATH = os.path.join(LIB_DIR, "libb200lmk.so")
HOST_SOURCE = os.path.join(CSRC, "host_torch.cpp")
HOST_PATH = os.path.join(LIB_DIR, "_lmk_host.so")
SOURCES = ["api.cu", "attn_general.cu", "attn_f32.cu", "attn_sm100.cu", "attn_mask_sm100.cu", "grouped_softmax.cu", "retrieval.cu",
           "scores_sm100.cu", "cache_store.cu", "decode.cu",
           "block_cache.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC"]


def _headers():
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))]
    return hs + [os.path.join(HERE, "..", "include", "b200lmk.h")]


def _newer(path, deps):
    if not os.path.exists(path):
        return True
    t = os.path.getmtime(path)
    return any(os.path.getmtime(d) > t for d in deps)


def _host_command():
    """g++ command line of the host layer, against the installed torch's headers and libraries."""
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"))
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
               os.path.join(cuda, "include"), sysconfig.get_path("include")]
    lib = os.path.join(root, "lib")
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", *["-isystem" + d for d in include], HOST_SOURCE, "-o", HOST_PATH,
            "-L" + lib, "-L" + os.path.join(cuda, "lib64"), "-Wl,-rpath," + lib, "-lc10", "-lc10_cuda", "-ltorch_cpu",
            "-ltorch_cuda", "-ltorch", "-ltorch_python", "-lcudart", "-ldl"]


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile the CUDA sources into landmark_attention_b200/lib/libb200lmk.so; returns the path."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    os.makedirs(LIB_DIR, exist_ok=True)
    os.makedirs(OBJ_DIR, exist_ok=True)
    headers = _headers()
    jobs = []
    for s in SOURCES:
        src, obj = os.path.join(CSRC, s), os.path.join(OBJ_DIR, s[:-3] + ".o")
        if force or _newer(obj, [src] + headers):
            cmd = [nvcc, *NVCC_FLAGS, "-c", src, "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append(cmd)
    n_objs = len(jobs)
    if force or _newer(HOST_PATH, [HOST_SOURCE] + headers):
        jobs.append(_host_command())
    objs = [os.path.join(OBJ_DIR, s[:-3] + ".o") for s in SOURCES]

    def run(cmd):
        return cmd, subprocess.run(cmd, capture_output=True, text=True)

    with ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as pool:
        for cmd, res in pool.map(run, jobs):
            if res.returncode != 0:
                raise RuntimeError("compiler failed: " + " ".join(cmd) + "\n" + res.stdout + res.stderr)
            if verbose:
                print(res.stderr)
    if n_objs or _newer(LIB_PATH, objs):
        res = subprocess.run([nvcc, "-shared", "-o", LIB_PATH, *objs], capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError("link failed:\n" + res.stdout + res.stderr)
    return LIB_PATH


if __name__ == "__main__":
    import sys
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
