"""Builds ``libnvfp4effma.so`` (the C-ABI shared library) in-tree from ``csrc/*.cu`` for sm_100a, and
``libnvfp4effma_torch-<version of torch>.so`` (the torch operators' CUDA kernels, host code that calls the C ABI) from ``csrc/torch_ops.cpp``.

    python -m nvfp4effma_b200.build [--force]

One nvcc process per translation unit, run in parallel, then one link step.  Objects live in ``csrc/_obj`` and are
rebuilt when a source or header is newer.  No GPU is needed: nvcc cross-compiles.
"""
import concurrent.futures
import glob
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(CSRC, "_obj")
LIB = os.path.join(HERE, "libnvfp4effma.so")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-O3", "-std=c++17", "-lineinfo", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC,-ffp-contract=off",
         "-Xptxas", "-v", "--expt-relaxed-constexpr"] + os.environ.get("NVFP4A_NVCC_FLAGS", "").split()


def _newest_header():
    hs = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(HERE, "..", "include", "*.h"))
    return max(os.path.getmtime(h) for h in hs)


def _compile(src, force):
    obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
    if not force and os.path.exists(obj) and os.path.getmtime(obj) > max(os.path.getmtime(src), _newest_header()):
        return obj, ""
    r = subprocess.run([NVCC, *FLAGS, "-c", "-o", obj, src], capture_output=True, text=True)
    if r.returncode:
        raise RuntimeError(f"nvcc failed on {src}:\n{r.stdout}\n{r.stderr}")
    return obj, r.stderr


def _build_torch(force):
    """The torch operators' library; its C-ABI calls resolve to LIB beside it."""
    src = os.path.join(CSRC, "torch_ops.cpp")
    newest = max(os.path.getmtime(f) for f in [src] + glob.glob(os.path.join(HERE, "..", "include", "*.h")))
    import torch
    out = os.path.join(HERE, f"libnvfp4effma_torch-{torch.__version__}.so")
    if not force and os.path.exists(out) and os.path.getmtime(out) > newest:
        return
    base = os.path.dirname(os.path.abspath(torch.__file__))
    cuda = os.path.dirname(os.path.dirname(NVCC))
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
                        f"-I{base}/include", f"-I{base}/include/torch/csrc/api/include", f"-I{cuda}/include", "-o", out, src,
                        f"-L{base}/lib", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda", f"-L{HERE}", "-lnvfp4effma", "-Wl,-rpath,$ORIGIN"],
                       capture_output=True, text=True)
    if r.returncode:
        raise RuntimeError(f"building {out} failed:\n{r.stdout}\n{r.stderr}")


def build(force=False, verbose=False):
    os.makedirs(OBJ, exist_ok=True)
    srcs = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        results = list(ex.map(lambda s: _compile(s, force), srcs))
    objs = [o for o, _ in results]
    log = "\n".join(l for _, l in results if l)
    if verbose and log:
        print(log)
    if force or not os.path.exists(LIB) or any(os.path.getmtime(o) > os.path.getmtime(LIB) for o in objs):
        r = subprocess.run([NVCC, "-shared", "-o", LIB, *objs, "-lcudart_static", "-ldl", "-lrt", "-lpthread"], capture_output=True, text=True)
        if r.returncode:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    _build_torch(force)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
