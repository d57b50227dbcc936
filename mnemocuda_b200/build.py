"""Build libmnemo_b200.so in-tree with nvcc for sm_100a (cross-compiles without a GPU).

    python -m mnemocuda_b200.build [--force] [--verbose]
"""
from __future__ import annotations

import glob
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libmnemo_b200.so")
NATIVE = os.path.join(HERE, "_native.so")  # Python binding of the library (csrc/binding.cpp)
BINDING = os.path.join(CSRC, "binding.cpp")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-lineinfo", "-std=c++17",
    "-Xcompiler", "-fPIC",
]
OBJ = os.path.join(HERE, "_obj")  # per-source objects (git-ignored): a change recompiles one file, in parallel with the rest


def sources() -> list[str]:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def needs_build() -> bool:
    if not os.path.exists(LIB) or not os.path.exists(NATIVE):
        return True
    if os.path.getmtime(BINDING) > os.path.getmtime(NATIVE):
        return True
    t = os.path.getmtime(LIB)
    deps = sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + [
        os.path.join(HERE, "..", "include", "mnemo_b200.h")]
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not needs_build():
        return LIB
    from concurrent.futures import ThreadPoolExecutor
    nvcc = os.environ.get("NVCC", "nvcc")
    env = dict(os.environ)
    env.pop("CC", None)
    env.pop("CXX", None)
    os.makedirs(OBJ, exist_ok=True)
    headers = glob.glob(os.path.join(CSRC, "*.cuh")) + [os.path.join(HERE, "..", "include", "mnemo_b200.h")]
    newest_header = max(os.path.getmtime(h) for h in headers)

    def compile_one(src: str) -> str:
        obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
        if force or not os.path.exists(obj) or os.path.getmtime(obj) < max(os.path.getmtime(src), newest_header):
            cmd = [nvcc, *NVCC_FLAGS, "-c", src, "-o", obj]
            if verbose:
                cmd += ["-Xptxas", "-v"]
            subprocess.check_call(cmd, env=env)
        return obj

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 2)) as pool:
        objs = list(pool.map(compile_one, sources()))
    subprocess.check_call([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-o", LIB, *objs, "-lcudart"],
                          env=env)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(shutil.which(nvcc) or "/usr/local/cuda/bin/nvcc")))
    subprocess.check_call([os.environ.get("HOST_CXX", "g++"), "-O2", "-std=c++20", "-fPIC", "-shared",
                           "-I" + os.path.join(cuda, "include"), "-I" + sysconfig.get_paths()["include"], BINDING, "-o", NATIVE,
                           "-L" + HERE, "-l:libmnemo_b200.so", "-L" + os.path.join(cuda, "lib64"), "-lcudart",
                           "-Wl,-rpath,$ORIGIN"], env=env)  # found beside the library, wherever the tree lies
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
