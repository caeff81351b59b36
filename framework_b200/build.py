"""Builds the native parts in-tree: ``libmni_b200.so`` with nvcc for sm_100a (cross-compiles without a GPU) and the
host extension ``_host.so`` (tensor object and operator front end) with g++ against torch's headers."""
from __future__ import annotations

import glob
import importlib.machinery
import importlib.util
import os
import subprocess
import sys

_PKG = os.path.dirname(os.path.abspath(__file__))
_ROOT = os.path.dirname(_PKG)
CSRC = os.path.join(_PKG, "csrc")
LIB_PATH = os.path.join(_PKG, "lib", "libmni_b200.so")
HOST_SRC = os.path.join(CSRC, "host", "host.cpp")
HOST_PATH = os.path.join(_PKG, "lib", "_host.so")

NVCC_FLAGS = [
    "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "-shared",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def sources() -> list:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def is_stale() -> bool:
    if not os.path.exists(LIB_PATH):
        return True
    t = os.path.getmtime(LIB_PATH)
    return any(os.path.getmtime(d) > t for d in sources() + _headers())


def source_hash() -> str:
    """sha256 over the names and contents of every file the library is built from."""
    import hashlib
    h = hashlib.sha256()
    for path in sorted(sources() + _headers()):
        h.update(os.path.basename(path).encode() + b"\0")
        with open(path, "rb") as f:
            h.update(f.read())
        h.update(b"\0")
    return h.hexdigest()


def _headers() -> list:
    return glob.glob(os.path.join(CSRC, "*.h")) + glob.glob(os.path.join(_ROOT, "include", "*.h"))


def build_library(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu under csrc/ (one nvcc per file, side by side; objects whose source and headers
    are unchanged are kept) and link them into lib/libmni_b200.so; returns its path."""
    if not force and not is_stale():
        return LIB_PATH
    os.makedirs(os.path.dirname(LIB_PATH), exist_ok=True)
    obj_dir = os.path.join(_PKG, "lib", "obj")
    os.makedirs(obj_dir, exist_ok=True)
    env = dict(os.environ)
    env.pop("CC", None)
    env.pop("CXX", None)
    compile_flags = [f for f in NVCC_FLAGS if f != "-shared"]
    newest_header = max((os.path.getmtime(h) for h in _headers()), default=0.0)
    jobs, objects = [], []
    for src in sources():
        obj = os.path.join(obj_dir, os.path.basename(src)[:-3] + ".o")
        objects.append(obj)
        fresh = (not force and os.path.exists(obj)
                 and os.path.getmtime(obj) >= max(os.path.getmtime(src), newest_header))
        if fresh:
            continue
        cmd = [_nvcc(), *compile_flags, "-I", os.path.join(_ROOT, "include"), "-I", CSRC]
        if verbose:
            cmd += ["-Xptxas", "-v"]
        cmd += ["-c", "-o", obj, src]
        jobs.append((src, subprocess.Popen(cmd, env=env)))
    # The hash of the sources is linked in, so that a loader can tell a library built from other sources.
    id_src, id_obj = os.path.join(obj_dir, "build_id.c"), os.path.join(obj_dir, "build_id.o")
    with open(id_src, "w") as f:
        f.write('__attribute__((visibility("default"))) const char *mni_b200_build_id(void) '
                '{ return "%s"; }\n' % source_hash())
    subprocess.check_call(["gcc", "-O1", "-fPIC", "-c", "-o", id_obj, id_src], env=env)
    failed = [src for src, proc in jobs if proc.wait() != 0]
    if failed:
        raise subprocess.CalledProcessError(1, f"nvcc -c {' '.join(failed)}")
    arch = NVCC_FLAGS[NVCC_FLAGS.index("-gencode"):NVCC_FLAGS.index("-gencode") + 2]
    subprocess.check_call([_nvcc(), *arch, "-shared", "-o", LIB_PATH, *objects, id_obj], env=env)
    return LIB_PATH


def host_source_hash() -> str:
    """sha256 of what the host extension is built from: its source, the C ABI header, the torch and Python versions."""
    import hashlib
    import torch
    h = hashlib.sha256(f"{torch.__version__} {sys.version_info[:3]}".encode())
    for path in [HOST_SRC] + sorted(glob.glob(os.path.join(_ROOT, "include", "*.h"))):
        with open(path, "rb") as f:
            h.update(f.read())
    return h.hexdigest()


def _hash_file() -> str:
    return HOST_PATH + ".id"


def host_is_stale() -> bool:
    try:
        with open(_hash_file()) as f:
            return f.read().strip() != host_source_hash() or not os.path.exists(HOST_PATH)
    except OSError:
        return True


def build_host(force: bool = False) -> str:
    """Compiles the host extension into lib/_host.so (about ten seconds); returns its path.  The file is put in place
    by a rename, so that whoever loads it meanwhile sees a whole one; of processes that find it missing at the same time
    (the ranks of a fresh tree) one compiles, under a file lock, and the others take what it has built."""
    if not force and not host_is_stale():
        return HOST_PATH
    import fcntl
    os.makedirs(os.path.dirname(HOST_PATH), exist_ok=True)
    with open(HOST_PATH + ".lock", "w") as lock:
        fcntl.flock(lock, fcntl.LOCK_EX)
        if force or host_is_stale():
            _compile_host()
    return HOST_PATH


def _compile_host() -> None:
    import sysconfig
    import torch
    root = os.path.dirname(torch.__file__)
    inc = [os.path.join(_ROOT, "include"), os.path.join(root, "include"),
           os.path.join(root, "include", "torch", "csrc", "api", "include"), sysconfig.get_paths()["include"],
           os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")]
    tmp = f"{HOST_PATH}.{os.getpid()}.tmp"
    subprocess.check_call(
        ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
         f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
         f'-DMNI_HOST_SOURCE_HASH="{host_source_hash()}"', *[f"-I{d}" for d in inc], HOST_SRC, "-o", tmp,
         "-L" + os.path.join(root, "lib"), "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10"])
    os.replace(tmp, HOST_PATH)
    with open(f"{tmp}.id", "w") as f:
        f.write(host_source_hash() + "\n")
    os.replace(f"{tmp}.id", _hash_file())


def load_host():
    """The host extension as a module, compiled first if it is missing or was built from another source."""
    import torch  # noqa: F401  (the extension links against torch's libraries, which torch loads)
    try:
        build_host()
    except (OSError, subprocess.CalledProcessError) as e:
        raise ImportError(f"{HOST_PATH} is missing or was built from another source, and cannot be built here ({e}): build it "
                          "with `python -m framework_b200.build`") from e
    loader = importlib.machinery.ExtensionFileLoader("_host", HOST_PATH)
    spec = importlib.util.spec_from_file_location("_host", HOST_PATH, loader=loader)
    module = importlib.util.module_from_spec(spec)
    loader.exec_module(module)
    if module.source_hash != host_source_hash():
        raise ImportError(f"{HOST_PATH} was built from another source than {HOST_SRC}; delete it and import again")
    return module


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
    print(build_host(force="--force" in sys.argv))
