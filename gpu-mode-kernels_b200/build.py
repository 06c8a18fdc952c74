"""Build liba2a.so (the C-ABI CUDA library, nvcc for sm_100a) and _host (the compiled part of the Python
layer, g++ against torch's headers) in-tree.

    python gpu-mode-kernels_b200/build.py [--verbose]

nvcc cross-compiles without a GPU.  The library links the CUDA runtime
statically, so it depends on nothing but the driver at run time.  _host depends on
the Python and the torch it was built against; its file name says which.
"""
import os
import shutil
import subprocess
import sys
import sysconfig

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG_DIR)
CSRC = os.path.join(PKG_DIR, "csrc")
LIB_PATH = os.path.join(PKG_DIR, "liba2a.so")
SOURCES = [os.path.join(CSRC, "a2a.cu"), os.path.join(CSRC, "a2a_noalloc.cu"), os.path.join(CSRC, "histogram.cu")]
HEADERS = [os.path.join(CSRC, "a2a_kernels.cuh"), os.path.join(CSRC, "a2a_pipe.cuh"), os.path.join(CSRC, "a2a_near.cuh"),
           os.path.join(CSRC, "a2a_solo.cuh"),
           os.path.join(CSRC, "a2a_device.cuh"),
           os.path.join(ROOT, "include", "a2a.h")]
HOST_SOURCE = os.path.join(CSRC, "host.cpp")


def nvcc_path() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found (set NVCC=/path/to/nvcc)")


def host_path() -> str:
    """Where _host for this Python and this torch lies: another one's is neither loaded nor taken for up to date."""
    import torch

    return os.path.join(PKG_DIR, f"_host.{sysconfig.get_config_var('SOABI')}.torch-{torch.__version__}.so")


def needs_build() -> bool:
    if not os.path.exists(LIB_PATH) or not os.path.exists(host_path()):
        return True
    t = min(os.path.getmtime(LIB_PATH), os.path.getmtime(host_path()))
    return any(os.path.getmtime(f) > t for f in SOURCES + HEADERS + [HOST_SOURCE, os.path.abspath(__file__)])


def run(tool: str, cmd, verbose: bool) -> None:
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"{tool} failed:\n" + " ".join(cmd) + "\n" + res.stdout + res.stderr)
    if verbose:
        print(res.stdout + res.stderr)


def build_host(verbose: bool = False) -> None:
    import torch

    torch_dir = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(nvcc_path())))
    include = [os.path.join(ROOT, "include"), os.path.join(torch_dir, "include"),
               os.path.join(torch_dir, "include", "torch", "csrc", "api", "include"), os.path.join(cuda, "include"),
               sysconfig.get_paths()["include"]]
    run("g++", [
        os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC",
        f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *("-I" + d for d in include), "-o", host_path(), HOST_SOURCE,
        "-L" + os.path.join(torch_dir, "lib"), "-ltorch_python", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda",
        "-L" + PKG_DIR, "-la2a", "-Wl,-rpath,$ORIGIN",
    ], verbose)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile both if one is missing or older than the sources; return the library's path."""
    if not force and not needs_build():
        return LIB_PATH
    cmd = [
        nvcc_path(), "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
        "-shared", "-Xcompiler", "-fPIC", "-cudart", "static",
        "-I", os.path.join(ROOT, "include"), "-I", CSRC,
        "-o", LIB_PATH, *SOURCES,
    ]
    if verbose:
        cmd[1:1] = ["-Xptxas", "-v"]
    run("nvcc", cmd, verbose)
    build_host(verbose)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force=True, verbose="--verbose" in sys.argv))
