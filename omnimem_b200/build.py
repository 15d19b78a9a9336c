"""Build recipe of the CUDA library (plain nvcc, sm_100a only) and of the native host path on top of it (g++ against
the installed torch); outputs in-tree.

    python -m omnimem_b200.build            # build if sources are newer than the library
    python -m omnimem_b200.build --force
"""
from __future__ import annotations

import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_PATH = os.path.join(HERE, "libomnimem_b200.so")
HOST_PATH = os.path.join(HERE, "_host.so")
SOURCES = ["capi.cu", "topk.cu", "sel_fwd.cu", "sel_fwd_tc.cu", "sel_bwd.cu", "cache.cu", "misc.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    cand = os.environ.get("NVCC") or os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    return cand if os.path.exists(cand) else "nvcc"


def sources() -> list[str]:
    extra = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu") and f not in SOURCES)
    return [os.path.join(CSRC, f) for f in SOURCES + extra]


def _stale() -> bool:
    if not (os.path.exists(LIB_PATH) and os.path.exists(HOST_PATH)):
        return True
    t = min(os.path.getmtime(LIB_PATH), os.path.getmtime(HOST_PATH))
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)]
    deps.append(os.path.join(os.path.dirname(HERE), "include", "omnimem_b200.h"))
    return any(os.path.getmtime(d) > t for d in deps)


def _host_commands(obj: str):
    """Compile and link commands of the native host path (csrc/host.cpp)."""
    import sysconfig

    from torch.utils import cpp_extension as ext
    cuda = os.path.dirname(os.path.dirname(_nvcc())) or "/usr/local/cuda"
    includes = [f"-I{p}" for p in (*ext.include_paths(), sysconfig.get_paths()["include"], os.path.join(cuda, "include"))]
    compile_ = ["g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_host",
                "-DTORCH_API_INCLUDE_EXTENSION_H", *includes, "-c", os.path.join(CSRC, "host.cpp"), "-o", obj]
    link = ["g++", "-shared", "-o", HOST_PATH, obj, f"-L{HERE}", "-l:" + os.path.basename(LIB_PATH), *(f"-L{p}" for p in ext.library_paths()),
            f"-L{os.path.join(cuda, 'lib64')}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python",
            "-lcudart", "-Wl,-rpath,$ORIGIN"]
    return compile_, link


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu under csrc/ into libomnimem_b200.so and host.cpp into _host.so (one compiler process
    per file, run in parallel, then the link steps).  Returns the library path."""
    if not force and not _stale():
        return LIB_PATH
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)
    procs = []
    host_obj = os.path.join(objdir, "host_cpp.o")
    host_compile, host_link = _host_commands(host_obj)
    host_src = os.path.join(CSRC, "host.cpp")
    deps = [host_src, os.path.join(os.path.dirname(HERE), "include", "omnimem_b200.h")]
    if force or not os.path.exists(host_obj) or any(os.path.getmtime(d) > os.path.getmtime(host_obj) for d in deps):
        procs.append((host_src, None, subprocess.Popen(host_compile, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for src in sources():
        obj = os.path.join(objdir, os.path.basename(src)[:-3] + ".o")
        cmd = [_nvcc(), *NVCC_FLAGS, "-c", src, "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
        procs.append((src, obj, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    objs = []
    for src, obj, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{out}")
        if verbose and out:
            print(out)
        if obj is not None:
            objs.append(obj)
    link = [_nvcc(), "-shared", "-o", LIB_PATH, *objs, "-lcudart"]
    for cmd in (link, host_link):
        r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}")
    return LIB_PATH


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
