"""Build recipe of the CUDA library (sm_100a only, in-tree output).

    python -m flashdp4review_b200.build            # build if sources are newer than the .so
    python -m flashdp4review_b200.build --force
"""
import os
import shutil
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB = os.path.join(PKG, "libfdp_b200.so")
HOST_LIB = os.path.join(PKG, "_fdp_host.so")
HOST_SOURCE = os.path.join(CSRC, "fdp_host.cpp")
SOURCES = ["fdp_abi.cu", "fdp_simt.cu", "fdp_layernorm.cu", "fdp_tc.cu", "fdp_static.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC"]


def _nvcc():
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC")


def sources():
    return [os.path.join(CSRC, s) for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]


def stale():
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if not f.endswith((".cpp", ".o"))]
    deps.append(os.path.join(os.path.dirname(PKG), "include", "fdp_b200.h"))
    return any(os.path.getmtime(d) > t for d in deps)


def build_host(force=False):
    """Compile the torch-facing call layer (csrc/fdp_host.cpp) into _fdp_host.so."""
    import sysconfig
    import torch
    from torch.utils import cpp_extension
    header = os.path.join(os.path.dirname(PKG), "include", "fdp_b200.h")
    tag = f"fdp_host for torch {torch.__version__}"      # the module carries it: another torch needs another build
    if not force and os.path.exists(HOST_LIB) and all(
            os.path.getmtime(d) <= os.path.getmtime(HOST_LIB) for d in (HOST_SOURCE, header)):
        with open(HOST_LIB, "rb") as f:
            if tag.encode() + b"\0" in f.read():
                return HOST_LIB
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    includes = cpp_extension.include_paths() + [sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-DTORCH_EXTENSION_NAME=_fdp_host",
           f'-DFDP_HOST_TAG="{tag}"',
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", HOST_SOURCE, "-o", HOST_LIB]
    cmd += ["-isystem" + d for d in includes]
    cmd += ["-L" + d for d in cpp_extension.library_paths()]
    cmd += ["-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"{cmd[0]} failed on {HOST_SOURCE}:\n{r.stderr}")
    return HOST_LIB


def build(force=False, verbose=False):
    """Compile every .cu of the package into libfdp_b200.so (one nvcc call per file, then link), and the
    call layer beside it."""
    build_host(force)
    if not force and not stale():
        return LIB
    nvcc = _nvcc()

    def compile_one(src):
        obj = src[:-3] + ".o"
        cmd = [nvcc] + NVCC_FLAGS + ["-c", src, "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        r = subprocess.run(cmd, capture_output=True, text=True)
        if verbose:
            sys.stderr.write(r.stderr)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{r.stderr}")
        return obj

    from concurrent.futures import ThreadPoolExecutor
    with ThreadPoolExecutor(max_workers=4) as ex:
        objs = list(ex.map(compile_one, sources()))
    r = subprocess.run([nvcc, "-shared", "-o", LIB] + objs, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stderr}")
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
