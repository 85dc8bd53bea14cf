"""Build libhqkv.so (the C-ABI library) in-tree with nvcc for sm_100a, and _host.so (the operators' host path, a CPython
module over it) with g++.

    python -m hqekv_b200.build          # rebuild if the library was not compiled from the sources present
    python -m hqekv_b200.build --force
    python -m hqekv_b200.build --checks # the bounds-check build, libhqkv_checked.so

Every build is stamped with a hash of its sources (hqkv_build_id()).

No --use_fast_math: the codec relies on IEEE division and explicit roundings.
"""
import hashlib
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
LIB_PATH = os.path.join(HERE, "libhqkv.so")
HOST_PATH = os.path.join(HERE, "_host.so")
SOURCES = ["codec.cu", "decode.cu", "flush.cu", "gemv.cu", "policy.cu"]
NVCC_FLAGS = [
    "-std=c++17", "-O3", "-lineinfo",
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def source_id():
    """First 16 hex digits of the SHA-256 over the library's sources (csrc sorted by name, then the header)."""
    h = hashlib.sha256()
    for path in sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC)) + [os.path.join(INCLUDE, "hqkv.h")]:
        with open(path, "rb") as f:
            h.update(os.path.basename(path).encode() + b"\0" + f.read())
    return h.hexdigest()[:16]


def library_id(path=LIB_PATH):
    """The stamp inside a built library, read from the file without loading it (None if there is none)."""
    marker = b"HQKV_BUILD_ID="
    try:
        with open(path, "rb") as f:
            blob = f.read()
    except OSError:
        return None
    at = blob.find(marker)
    if at < 0:
        return None
    end = blob.find(b"\0", at)
    return blob[at + len(marker):end].decode(errors="replace")


def needs_build():
    """True when the library or the host module is missing or was compiled from other sources than the ones present."""
    return library_id(LIB_PATH) != source_id() or library_id(HOST_PATH) != source_id()


CHECKED_LIB_PATH = os.path.join(HERE, "libhqkv_checked.so")


def build(force=False, verbose=False, checks=False):
    """Compile every .cu into objects and link the shared library.  Returns its path.
    ``checks``: the bounds-check build (-DHQKV_CHECKS) into libhqkv_checked.so; load it with HQKV_LIB=<path>."""
    if os.environ.get("HQKV_LIB") and not checks:
        return os.environ["HQKV_LIB"]  # the caller points at a library it built itself
    if checks:
        if not force and os.path.exists(CHECKED_LIB_PATH) and library_id(CHECKED_LIB_PATH) == source_id():
            return CHECKED_LIB_PATH
        return _compile(CHECKED_LIB_PATH, os.path.join(HERE, "build", "checked"), ["-DHQKV_CHECKS"], verbose)
    if not force and not needs_build():
        return LIB_PATH
    host = _compile_host()
    path = _compile(LIB_PATH, os.path.join(HERE, "build"), [], verbose)
    out, _ = host.communicate()
    if host.returncode != 0:
        raise RuntimeError(f"g++ failed on host.cpp:\n{out}")
    return path


def _compile_host():
    """Start the compiler on the host module; torch's headers and libraries are those of the running interpreter."""
    import sysconfig
    import torch
    root = os.path.join(os.path.dirname(torch.__file__))
    cuda = os.path.dirname(os.path.dirname(_nvcc())) if os.path.isabs(_nvcc()) else "/usr/local/cuda"
    cmd = ["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DHQKV_BUILD_ID="{source_id()}"',
           "-I", INCLUDE, "-I", os.path.join(root, "include"), "-I", os.path.join(cuda, "include"),
           "-I", sysconfig.get_paths()["include"], os.path.join(CSRC, "host.cpp"), "-o", HOST_PATH,
           "-L", os.path.join(root, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python",
           "-Wl,-rpath," + os.path.join(root, "lib")]
    return subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)


def _compile(lib_path, objdir, extra, verbose):
    os.makedirs(objdir, exist_ok=True)
    nvcc = _nvcc()
    extra = [*extra, f'-DHQKV_BUILD_ID="{source_id()}"']
    procs = []
    for src in SOURCES:
        obj = os.path.join(objdir, src.replace(".cu", ".o"))
        cmd = [nvcc, *NVCC_FLAGS, *extra, "-I", INCLUDE, "-I", CSRC, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append((src, obj, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    objs = []
    for src, obj, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{out}")
        if verbose and out:
            print(out)
        objs.append(obj)
    link = [nvcc, "-shared", "-o", lib_path, *objs, "-Xcompiler", "-fPIC"]  # static cudart (nvcc default)
    r = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}")
    return lib_path


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="-v" in sys.argv, checks="--checks" in sys.argv)
    print(path)
