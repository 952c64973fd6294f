"""Build recipe of the native library: ``python -m fovi_b200.build``.

Compiles ``fovi_b200/csrc/*.cu`` with nvcc for sm_100a (one object per source, in parallel, only the
stale ones) and links them into ``fovi_b200/libfovi_b200.so``; ``csrc/bind.cpp``, the launch path for torch
tensors, becomes the extension module ``fovi_b200/_native<suffix of the interpreter>.so`` (both in-tree; objects and shared objects are
not committed).  The module is for one interpreter and one torch: its file name says the one, a stamp beside it and the
module itself the other.  Where it cannot be compiled the package runs on its Python path, and says so.
"""
import os
import importlib.util
import subprocess
import sys
import sysconfig
import warnings
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(CSRC, "build")
LIB = os.path.join(HERE, "libfovi_b200.so")
NATIVE = os.path.join(HERE, "_native" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))
SOURCES = ["capi.cu", "sampler.cu", "knnconv.cu", "knnconv_tc.cu", "knnconv_tc2.cu", "knnconv_tcp.cu", "knnpool.cu", "knnnorm.cu", "blocktrain.cu", "fused.cu", "tables.cu", "geometry.cu", "grad.cu", "knnconv_dw.cu", "depthwise.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC"]


def _headers_mtime():
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hs.append(os.path.join(HERE, "..", "include", "fovi_b200.h"))
    hs.append(os.path.abspath(__file__))
    return max(os.path.getmtime(h) for h in hs)


def _torch_version():
    """(folder of the installed torch, its version), without importing it."""
    folder = importlib.util.find_spec("torch").submodule_search_locations[0]
    scope = {}
    with open(os.path.join(folder, "version.py")) as f:
        exec(f.read(), scope)
    return folder, str(scope["__version__"])


def build_native(force=False):
    """The extension module of the launch path, against the interpreter and the torch that are installed.  Returns its path, or None, with a warning, where it cannot
    be compiled (no compiler, no headers): a module that was there is removed then, and the package runs without."""
    src, stamp = os.path.join(CSRC, "bind.cpp"), os.path.splitext(NATIVE)[0] + ".stamp"
    torch, version = _torch_version()
    made_for = f"torch {version}, python {sys.version}"
    newest = max(os.path.getmtime(f) for f in (src, os.path.join(HERE, "..", "include", "fovi_b200.h"), os.path.abspath(__file__)))
    plain = os.path.join(os.path.dirname(NATIVE), "_native.so")          # a name that any interpreter would import
    if plain != NATIVE and os.path.exists(plain):
        os.remove(plain)
    if not force and os.path.exists(NATIVE) and os.path.getmtime(NATIVE) >= newest and os.path.exists(stamp):
        with open(stamp) as f:
            if f.read() == made_for:
                return NATIVE
    fresh = f"{NATIVE}.{os.getpid()}"                                     # in one piece, or not at all, for a process that imports it meanwhile
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", f'-DFOVI_TORCH_VERSION="{version}"', f"-I{torch}/include",
           f"-I{torch}/include/torch/csrc/api/include", "-I" + sysconfig.get_paths()["include"], src, "-o", fresh, f"-L{torch}/lib", "-lc10", "-ltorch_cpu",
           "-ltorch_python"]
    try:
        r = subprocess.run(cmd, capture_output=True, text=True)
        failed = r.stdout + r.stderr if r.returncode else None
    except OSError as e:
        failed = str(e)
    for f in [stamp] + ([fresh, NATIVE] if failed else []):
        if os.path.exists(f):
            os.remove(f)
    if failed:
        warnings.warn(f"csrc/bind.cpp was not compiled; fovi_b200 launches its kernels from Python, which is slower:\n{failed}")
        return None
    os.replace(fresh, NATIVE)
    with open(stamp, "w") as f:
        f.write(made_for)
    return NATIVE


def build(force=False, verbose=False, defines=(), lib=None, obj_dir=None):
    """Compile what is stale and link.  `defines` ("NAME=value" strings), `lib` and `obj_dir` give a variant
    build beside the default one.  Returns the path of the shared object."""
    lib = lib or LIB
    obj_dir = obj_dir or OBJ
    os.makedirs(obj_dir, exist_ok=True)
    nvcc = os.environ.get("NVCC", "nvcc")
    hdr_t = _headers_mtime()
    flags = NVCC_FLAGS + [f"-D{d}" for d in defines] + (["-Xptxas", "-v"] if verbose else [])
    jobs = []
    for s in SOURCES:
        src, obj = os.path.join(CSRC, s), os.path.join(obj_dir, s[:-3] + ".o")
        if force or not os.path.exists(obj) or os.path.getmtime(obj) < max(os.path.getmtime(src), hdr_t):
            jobs.append((s, [nvcc] + flags + ["-c", src, "-o", obj]))

    def run(job):
        return job[0], subprocess.run(job[1], capture_output=True, text=True)

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as pool:
        for name, r in pool.map(run, jobs):
            if verbose or r.returncode:
                sys.stderr.write(r.stdout + r.stderr)
            if r.returncode:
                raise RuntimeError(f"nvcc failed on {name}")
    objs = [os.path.join(obj_dir, s[:-3] + ".o") for s in SOURCES]
    if jobs or not os.path.exists(lib) or os.path.getmtime(lib) < max(os.path.getmtime(o) for o in objs):
        r = subprocess.run([nvcc] + NVCC_FLAGS[:2] + ["-shared", "-o", lib] + objs, capture_output=True, text=True)
        if r.returncode:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("linking libfovi_b200.so failed")
    if lib == LIB:
        build_native(force)
    return lib


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
