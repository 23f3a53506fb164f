"""In-tree build: ``python -m linquant_b200.build`` -> linquant_b200/liblinquant_b200.so and linquant_b200/_host.so.

The CUDA library is plain nvcc for sm_100a with a C ABI; it links against the CUDA runtime only (no torch headers).
``_host`` is the CPython module that hands torch tensors to the library's whole-call entries (g++, torch headers)."""

from __future__ import annotations

import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "csrc", "build")
LIB = os.path.join(HERE, "liblinquant_b200.so")
HOST_SRC = os.path.join(CSRC, "host", "lq_host.cpp")
HOST_LIB = os.path.join(HERE, "_host.so")
HOST_KEY = os.path.join(OBJ, "lq_host.key")  # what the object of _host was compiled for
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
# no fast-math: precise division / sqrt / expf are required by the code rule
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-Xptxas", "-v"]


def sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _stale(src, obj):
    if not os.path.exists(obj):
        return True
    t = os.path.getmtime(obj)
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cuh")]
    deps += [os.path.join(CSRC, src), os.path.join(HERE, "..", "include", "linquant_b200.h")]
    return any(os.path.getmtime(d) > t for d in deps)


def _compile(src):
    obj = os.path.join(OBJ, src[:-3] + ".o")
    if not _stale(src, obj):
        return src, ""
    r = subprocess.run([NVCC, *FLAGS, "-c", os.path.join(CSRC, src), "-o", obj], capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed on {src}:\n{r.stdout}\n{r.stderr}")
    with open(obj[:-2] + ".ptxas", "w") as f:  # registers, spills and shared memory of every kernel
        f.write(r.stderr)
    return src, r.stderr


def host_key():
    """The ABI that ``_host`` is tied to; ``_cabi.host()`` compares it with the running one."""
    import torch

    return f"torch {torch.__version__}, {sysconfig.get_config_var('SOABI')}"


def _host_stale(obj):
    if _stale(os.path.join("host", "lq_host.cpp"), obj) or not os.path.exists(HOST_KEY):
        return True
    with open(HOST_KEY) as f:
        return f.read() != host_key()


def _compile_host(_=None):
    """The object file of ``_host``, and the torch library directories to link it against."""
    from torch.utils import cpp_extension as ext

    obj = os.path.join(OBJ, "lq_host.o")
    if _host_stale(obj):
        inc = ext.include_paths() + [sysconfig.get_paths()["include"], "/usr/local/cuda/include"]
        cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-Wall", f'-DLQ_BUILT_FOR="{host_key()}"', *[a for i in inc for a in ("-isystem", i)],
               "-c", HOST_SRC, "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"g++ failed on lq_host.cpp:\n{r.stdout}\n{r.stderr}")
        with open(HOST_KEY, "w") as f:
            f.write(host_key())
    return obj, ext.library_paths()


def build(verbose=False):
    os.makedirs(OBJ, exist_ok=True)
    with ThreadPoolExecutor(max_workers=os.cpu_count() or 4) as ex:
        host = ex.submit(_compile_host)
        logs = list(ex.map(_compile, sources()))
        host_obj, torch_libs = host.result()
    objs = [os.path.join(OBJ, s[:-3] + ".o") for s in sources()]
    if (not os.path.exists(LIB)) or any(os.path.getmtime(o) > os.path.getmtime(LIB) for o in objs):
        r = subprocess.run([NVCC, "-shared", "-o", LIB, *objs, "-lcudart"], capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    if (not os.path.exists(HOST_LIB)) or any(os.path.getmtime(o) > os.path.getmtime(HOST_LIB) for o in (host_obj, LIB)):
        r = subprocess.run(["g++", "-shared", "-o", HOST_LIB, host_obj, f"-L{HERE}", "-llinquant_b200", *[f"-L{d}" for d in torch_libs], "-ltorch_python",
                            "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda", "-Wl,-rpath,$ORIGIN"],
                           capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link of _host failed:\n{r.stdout}\n{r.stderr}")
    if verbose:
        for s, log in logs:
            if log:
                print(f"==== {s}\n{log}")
    return LIB


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv))
