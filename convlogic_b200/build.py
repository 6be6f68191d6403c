"""Build the native code in-tree: ``python -m convlogic_b200.build``.

Every ``csrc/*.cu`` is compiled for sm_100a with nvcc and linked into
``csrc/libconvlogic_b200.so`` (a plain C-ABI shared library, no torch or Python headers);
``csrc/torch_bind.cpp`` becomes ``csrc/_clb_torch.so``, the torch extension module over it.
"""

import glob
import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "csrc")
LIB = os.path.join(CSRC, "libconvlogic_b200.so")
BIND = os.path.join(CSRC, "_clb_torch.so")
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
FLAGS = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC", "--use_fast_math=false"]


def _nvcc():
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; the CUDA library cannot be built")
    return exe


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force=False, verbose=False, extra=()):
    nvcc = _nvcc()
    headers = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(
        os.path.join(os.path.dirname(CSRC), "..", "include", "*.h"))
    flags = [f for f in FLAGS if not f.startswith("--use_fast_math")] + list(extra)
    objs = []

    def compile_one(src):
        obj = src[:-3] + ".o"
        if force or _stale(obj, [src] + headers):
            cmd = [nvcc, *ARCH, *flags, "-c", src, "-o", obj]
            if verbose:
                print(" ".join(cmd), flush=True)
            r = subprocess.run(cmd, capture_output=True, text=True)
            if r.returncode:
                raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
            if verbose and (r.stdout or r.stderr):
                print(r.stdout, r.stderr)
        return obj

    def compile_binding():
        src, obj = BIND[:-len("_clb_torch.so")] + "torch_bind.cpp", BIND[:-3] + ".o"
        if force or _stale(obj, [src] + headers):
            import torch

            root = os.path.dirname(torch.__file__)
            inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
                   os.path.join(os.path.dirname(os.path.dirname(nvcc)), "include"), sysconfig.get_paths()["include"]]
            cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-DTORCH_EXTENSION_NAME=_clb_torch",
                   f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *[f"-I{d}" for d in inc], "-c", src, "-o", obj]
            r = subprocess.run(cmd, capture_output=True, text=True)
            if r.returncode:
                raise RuntimeError(f"g++ failed for {src}:\n{r.stdout}\n{r.stderr}")
        return obj

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as ex:
        bind_obj = ex.submit(compile_binding)
        objs = list(ex.map(compile_one, sources()))
        bind_obj = bind_obj.result()
    if force or _stale(LIB, objs):
        cmd = [nvcc, *ARCH, "-shared", "-o", LIB, *objs]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    if force or _stale(BIND, [bind_obj, LIB]):
        import torch

        lib_dir = os.path.join(os.path.dirname(torch.__file__), "lib")
        cmd = ["g++", "-shared", "-o", BIND, bind_obj, f"-L{lib_dir}", "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_cuda",
               "-ltorch_python", f"-L{CSRC}", "-l:libconvlogic_b200.so", "-Wl,-rpath,$ORIGIN"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True,
                extra=["-Xptxas", "-v"] if "--ptxas" in sys.argv else ()))
