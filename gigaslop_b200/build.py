"""Build recipe for libgigaslop_b200.so (nvcc, sm_100a only) and _native.so (g++), both in-tree."""
import os
import shutil
import subprocess

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
LIB = os.path.join(PKG, "libgigaslop_b200.so")
PTXAS_LOG = os.path.join(PKG, "libgigaslop_b200.ptxas.txt")    # ptxas -v of the last build: registers and spills per kernel
SRC = os.path.join(PKG, "csrc", "lib.cu")
NATIVE = os.path.join(PKG, "_native.so")                       # native call path of the Python operators
NATIVE_SRC = os.path.join(PKG, "csrc", "binding.cpp")
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3", "-lineinfo",
              "-shared", "-Xcompiler", "-fPIC", "-Xptxas=-v"]


def _nvcc():
    for cand in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; libgigaslop_b200.so cannot be built")


def sources():
    d = os.path.join(PKG, "csrc")
    inc = os.path.join(ROOT, "include", "gigaslop_b200")
    out = [os.path.join(d, f) for f in sorted(os.listdir(d)) if not f.endswith(".cpp")]
    for base, _, files in os.walk(inc):
        out += [os.path.join(base, f) for f in files]
    return out


def is_stale():
    if not os.path.exists(LIB) or not os.path.exists(PTXAS_LOG):
        return True
    t = os.path.getmtime(LIB)
    return any(os.path.getmtime(s) > t for s in sources())


def build(force=False, verbose=False, defines=(), out=None):
    """Compile the CUDA library if missing or older than its sources.  The resource report of ptxas (registers,
    spill bytes per kernel) is kept beside the library; ``kernel_resources()`` parses it.  ``defines`` / ``out``
    build a variant (``-DGSB200_DIAG`` for the tuning diagnostics) somewhere else."""
    target = out or LIB
    if out is None:
        build_native(force)
    if out is None and not force and not is_stale():
        return LIB
    cmd = [_nvcc(), *NVCC_FLAGS, *["-D" + d for d in defines], "-I" + os.path.join(ROOT, "include"), "-o", target, SRC]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + r.stdout[-4000:])
    with open(PTXAS_LOG if out is None else target + ".ptxas.txt", "w") as f:
        f.write(r.stdout)
    if verbose:
        print(r.stdout)
    return target


def native_target():
    """What _native.so is built for: it looks into torch's tensors, whose layout belongs to a release (and a C++ ABI) of torch."""
    import platform
    import torch
    return f"torch {torch.__version__}, C++11 ABI {int(torch._C._GLIBCXX_USE_CXX11_ABI)}, Python {platform.python_version()}"


def native_is_stale():
    """_native.so is missing, older than its sources, or built for another torch or Python (the text it carries says which)."""
    deps = [NATIVE_SRC, os.path.join(ROOT, "include", "gigaslop_b200", "gigaslop_b200.h")]
    if not os.path.exists(NATIVE) or any(os.path.getmtime(f) > os.path.getmtime(NATIVE) for f in deps):
        return True
    with open(NATIVE, "rb") as f:
        return native_target().encode() + b"\0" not in f.read()


def build_native(force=False):
    """Compile _native.so (CPython extension on torch's C++ headers) if it is stale."""
    if not force and not native_is_stale():
        return NATIVE
    import sysconfig
    import torch
    t = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    inc = [sysconfig.get_paths()["include"], os.path.join(ROOT, "include"), os.path.join(t, "include"),
           os.path.join(t, "include", "torch", "csrc", "api", "include"), os.path.join(cuda, "include")]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DGSB200_NATIVE_TARGET="{native_target()}"', *["-I" + i for i in inc], "-o", NATIVE, NATIVE_SRC,
           "-L" + os.path.join(t, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python"]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError("compiling the native binding failed:\n" + r.stdout[-4000:])
    return NATIVE


def kernel_resources(log=None):
    """{mangled kernel name: dict(registers, stack, spill_stores, spill_loads)} from the ptxas report of the build."""
    import re
    text = open(log or PTXAS_LOG).read()
    out = {}
    for block in re.split(r"ptxas info\s+: Compiling entry function '", text)[1:]:
        name = block.split("'")[0]
        sp = re.search(r"(\d+) bytes stack frame, (\d+) bytes spill stores, (\d+) bytes spill loads", block)
        rg = re.search(r"Used (\d+) registers", block)
        if sp and rg:
            out[name] = dict(registers=int(rg.group(1)), stack=int(sp.group(1)), spill_stores=int(sp.group(2)),
                             spill_loads=int(sp.group(3)))
    return out


if __name__ == "__main__":
    import sys
    print(build(force=True, verbose="-v" in sys.argv))
