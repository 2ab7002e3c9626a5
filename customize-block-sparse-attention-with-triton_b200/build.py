"""Builds libbsattn.so (the C-ABI CUDA library, nvcc for sm_100a) and _native.so (the host path of the
public op, a torch extension module linked to it) in-tree.

Usage:  python build.py [--force] [--verbose]
Both land next to the Python host layer (fa2_custom_mask/).
"""
import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "fa2_custom_mask", "libbsattn.so")
NATIVE_SRC = os.path.join(CSRC, "native.cpp")
NATIVE_OUT = os.path.join(HERE, "fa2_custom_mask", "_native.so")

NVCC_FLAGS = [
    "-std=c++17", "-O3", "-lineinfo",
    "-gencode", "arch=compute_100a,code=sm_100a",
    "--shared", "-Xcompiler", "-fPIC",
    "-cudart", "shared",
]


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _digest(files, flags):
    h = hashlib.sha256()
    for f in sorted(files) + [os.path.join(HERE, "..", "include", "bsattn.h")]:
        with open(f, "rb") as fh:
            h.update(os.path.basename(f).encode())
            h.update(fh.read())
    h.update(" ".join(flags).encode())
    return h.hexdigest()


def _compile(out, digest, cmd, force, verbose):
    """Runs cmd to make out; skipped when out was made from the same sources and flags."""
    stamp = out + ".stamp"
    if not force and os.path.exists(out) and os.path.exists(stamp):
        with open(stamp) as fh:
            if fh.read().strip() == digest:
                return
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or proc.returncode != 0:
        sys.stderr.write(proc.stdout + proc.stderr)
    if proc.returncode != 0:
        raise RuntimeError(f"{os.path.basename(cmd[0])} failed building {os.path.basename(out)}")
    with open(stamp, "w") as fh:
        fh.write(digest)


def find_nvcc():
    cand = shutil.which("nvcc") or os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found; libbsattn.so cannot be built")
    return cand


def _native_command():
    """g++ for the torch extension module; torch's own libraries are loaded by `import torch`, the C-ABI
    library is found beside the module."""
    import torch
    from torch.utils import cpp_extension
    dirs = cpp_extension.include_paths() + [sysconfig.get_paths()["include"],
                                            os.path.join(os.path.dirname(os.path.dirname(find_nvcc())), "include")]
    lib_dir = os.path.join(os.path.dirname(torch.__file__), "lib")
    return (["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden",
             f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"]
            + [f"-I{d}" for d in dirs] + [NATIVE_SRC, "-o", NATIVE_OUT, f"-L{lib_dir}"]
            + ["-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-lc10", "-lc10_cuda"]
            + [f"-L{os.path.dirname(OUT)}", "-l:libbsattn.so", "-Wl,-rpath,$ORIGIN"])


def build(force=False, verbose=False):
    """Compiles every .cu under csrc/ into one shared library and native.cpp into the module beside it;
    each is skipped when its sources are unchanged."""
    files = [os.path.join(CSRC, f) for f in os.listdir(CSRC)]
    cmd = [find_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + sources() + ["-o", OUT]
    _compile(OUT, _digest([f for f in files if f != NATIVE_SRC], NVCC_FLAGS), cmd, force, verbose)
    import torch
    native = _native_command()
    flags = [a for a in native if os.sep not in a] + [torch.__version__]  # no paths: the tree may move
    _compile(NATIVE_OUT, _digest([NATIVE_SRC], flags), native, force, verbose)
    return OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
