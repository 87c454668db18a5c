"""In-tree build of the CUDA library (nvcc, sm_100a only) and of the torch host module.

``build()`` compiles every ``csrc/*.cu`` into ``lib/libflexgemm_b200.so`` and
``csrc/host/fgb_torch.cpp`` (g++, against torch's headers) into
``lib/_fgb_torch.<python>.torch<version>.so`` next to the package, so the binaries
travel with a copy of the source tree.  It is incremental: a file is rebuilt only
when its source or a header is newer; a host module built for another Python or
torch has another name and is never loaded.
"""
import os
import shutil
import subprocess

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
INCLUDE = os.path.join(os.path.dirname(PKG), "include")
LIB_DIR = os.path.join(PKG, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libflexgemm_b200.so")
OBJ_DIR = os.path.join(LIB_DIR, "obj")
HOST_SRC = os.path.join(CSRC, "host", "fgb_torch.cpp")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]


def _nvcc():
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: the flexgemm_b200 CUDA library cannot be built")


def _newest(paths):
    return max(os.path.getmtime(p) for p in paths)


def host_path() -> str:
    """The host module of this Python and this torch: it is bound to the ABI of both."""
    import sysconfig
    import torch
    return os.path.join(LIB_DIR, f"_fgb_torch.{sysconfig.get_config_var('SOABI')}.torch{torch.__version__}.so")


def _build_host(force: bool):
    """Command and process of the torch host module's build, or None when it is up to date."""
    path = host_path()
    newest = _newest([HOST_SRC] + [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE) if f.endswith(".h")])
    if not force and os.path.exists(path) and os.path.getmtime(path) >= newest:
        return None
    import sysconfig
    import torch
    tdir = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    cmd = [os.environ.get("CXX", "g++"), "-shared", "-fPIC", "-O2", "-std=c++17",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-I" + os.path.join(tdir, "include"), "-I" + os.path.join(tdir, "include", "torch", "csrc", "api", "include"),
           "-I" + os.path.join(cuda, "include"), "-I" + sysconfig.get_path("include"), HOST_SRC, "-o", path,
           "-L" + os.path.join(tdir, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python",
           "-L" + os.path.join(cuda, "lib64"), "-lcudart"]
    return cmd, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)


def build(force: bool = False, verbose: bool = False) -> str:
    nvcc = _nvcc()
    os.makedirs(OBJ_DIR, exist_ok=True)
    sources = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers += [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE) if f.endswith(".h")]
    hdr_time = _newest(headers)
    objs, rebuilt = [], False
    procs = []
    host = _build_host(force)
    for src in sources:
        s = os.path.join(CSRC, src)
        o = os.path.join(OBJ_DIR, src[:-3] + ".o")
        objs.append(o)
        if force or not os.path.exists(o) or os.path.getmtime(o) < max(os.path.getmtime(s), hdr_time):
            cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", s, "-o", o]
            procs.append((cmd, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
            rebuilt = True
    for cmd, p in procs:
        out, _ = p.communicate()
        if verbose and out:
            print(out)
        if p.returncode != 0:
            raise RuntimeError("nvcc failed: %s\n%s" % (" ".join(cmd), out))
    if rebuilt or not os.path.exists(LIB_PATH):
        cmd = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB_PATH] + objs
        r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        if r.returncode != 0:
            raise RuntimeError("link failed: %s\n%s" % (" ".join(cmd), r.stdout))
    if host is not None:
        out, _ = host[1].communicate()
        if host[1].returncode != 0:
            raise RuntimeError("host module build failed: %s\n%s" % (" ".join(host[0]), out))
    return LIB_PATH


if __name__ == "__main__":
    import sys
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
