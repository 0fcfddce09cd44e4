"""Builds libgoph_b200.so in-tree with nvcc for sm_100a.

Each csrc/*.cu is compiled to an object (in parallel, skipped when up to date) and the
objects are linked into one shared library with the CUDA runtime linked statically, so the
library has no toolkit dependency at run time beyond the driver.
"""
import os
import platform
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
# GOPH_TUNING=1 builds a second library with the kernels' cycle probes compiled in (tuning only;
# nothing in the package loads it unless GOPH_B200_LIB points at it)
TUNING = os.environ.get("GOPH_TUNING") == "1"
OBJ = os.path.join(HERE, "build_tuning" if TUNING else "build")
LIB = os.path.join(HERE, "libgoph_b200_tuning.so" if TUNING else "libgoph_b200.so")
# the caller of the C ABI that runtime.py uses, for this Python (the suffix names its version and machine)
PYCALL = os.path.join(HERE, "goph_pycall" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))

NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
         "-Xcompiler", "-fPIC,-fvisibility=hidden", "--use_fast_math=false"]
FLAGS = [f for f in FLAGS if f != "--use_fast_math=false"]  # precise math only
if TUNING:
    FLAGS.append("-DGOPH_TUNING")
    if os.environ.get("GOPH_SPIN_NS"):
        FLAGS.append("-DGOPH_SPIN_NS=" + os.environ["GOPH_SPIN_NS"])
        OBJ += "_spin"
        LIB = LIB.replace("_tuning", "_tuning_spin")


def _sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _deps_mtime():
    hdrs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hdrs.append(os.path.join(HERE, "..", "include", "goph_b200.h"))
    return max(os.path.getmtime(h) for h in hdrs)


def _compile(src, verbose):
    obj = os.path.join(OBJ, src[:-3] + ".o")
    path = os.path.join(CSRC, src)
    if os.path.exists(obj) and os.path.getmtime(obj) >= max(os.path.getmtime(path), _deps_mtime()):
        return obj, False
    cmd = [NVCC, *FLAGS, "-c", path, "-o", obj]
    if verbose:
        cmd.insert(1, "-Xptxas=-v")
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("nvcc failed for %s:\n%s\n%s" % (src, r.stdout, r.stderr))
    if verbose:
        sys.stderr.write(r.stderr)
    return obj, True


def _pycall_wanted():
    """runtime.py does without the module (through ctypes, slower) where it cannot be: another machine, no Python headers."""
    return platform.machine() in ("x86_64", "AMD64") and os.name == "posix" and os.path.exists(
        os.path.join(sysconfig.get_paths()["include"], "Python.h"))


def _build_pycall(force):
    src = os.path.join(CSRC, "pycall.c")
    if not _pycall_wanted():
        return
    if not force and os.path.exists(PYCALL) and os.path.getmtime(PYCALL) >= os.path.getmtime(src):
        return
    cmd = [os.environ.get("CC", "gcc"), "-O2", "-shared", "-fPIC", "-I", sysconfig.get_paths()["include"], src, "-o", PYCALL]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("gcc failed for pycall.c:\n%s\n%s" % (r.stdout, r.stderr))


def build(force=False, verbose=False):
    _build_pycall(force)
    os.makedirs(OBJ, exist_ok=True)
    if force:
        for f in os.listdir(OBJ):
            if f.endswith(".o"):
                os.remove(os.path.join(OBJ, f))
    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as ex:
        results = list(ex.map(lambda s: _compile(s, verbose), _sources()))
    objs = [o for o, _ in results]
    if any(changed for _, changed in results) or not os.path.exists(LIB):
        cmd = [NVCC, "-shared", "-cudart", "static", "-gencode", "arch=compute_100a,code=sm_100a",
               "-o", LIB, *objs, "-ldl"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("link failed:\n%s\n%s" % (r.stdout, r.stderr))
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
