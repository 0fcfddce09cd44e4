"""The caller of the C ABI (csrc/pycall.c) and what stands in for it, on functions compiled here; no GPU."""
import ctypes as C
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

ECHO = """
#include <stdint.h>
uint64_t seen_w[18]; float seen_f[2];
int echo(const void* a, uint64_t b, int c, float d, void* e, const int* f, int g, float h, void* i, uint64_t j, int k, void* l) {
  seen_w[0] = (uint64_t)a; seen_w[1] = b; seen_w[2] = (uint64_t)(int64_t)c; seen_f[0] = d; seen_w[4] = (uint64_t)e;
  seen_w[5] = f ? (uint64_t)*f : 77; seen_w[6] = (uint64_t)(int64_t)g; seen_f[1] = h; seen_w[8] = (uint64_t)i; seen_w[9] = j;
  seen_w[10] = (uint64_t)(int64_t)k; seen_w[11] = (uint64_t)l;
  return c - 3;
}
"""


@pytest.fixture(scope="module")
def echo(tmp_path_factory):
    d = tmp_path_factory.mktemp("echo")
    (d / "echo.c").write_text(ECHO)
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", str(d / "echo.c"), "-o", str(d / "echo.so")], check=True)
    return C.CDLL(str(d / "echo.so"))


def _callers(pkg, lib):
    """Both ways a per-step entry point is called."""
    sig = "pnifppifpnip"
    mod = pkg.runtime._pycall()
    if mod is not None:
        yield mod.Function(C.cast(lib.echo, C.c_void_p).value, sig)
    f = C.CFUNCTYPE(C.c_int, *[pkg.runtime._CTYPES[k] for k in sig])
    yield f(C.cast(lib.echo, C.c_void_p).value)


def test_arguments_arrive(pkg, echo):
    words, floats = (C.c_uint64 * 18).in_dll(echo, "seen_w"), (C.c_float * 2).in_dll(echo, "seen_f")
    for call in _callers(pkg, echo):
        assert call(1 << 40, (1 << 63) + 5, -7, 0.5, None, (C.c_int * 1)(31), 2, -1e-6, C.c_void_p(9), 0, -1, 1 << 63) == -10
        assert [words[i] for i in (0, 1, 4, 5, 6, 8, 9, 11)] == [1 << 40, (1 << 63) + 5, 0, 31, 2, 9, 0, 1 << 63]
        assert [C.c_int64(words[i]).value for i in (2, 10)] == [-7, -1]
        assert floats[0] == 0.5 and floats[1] == C.c_float(-1e-6).value


def test_wrong_arguments_raise(pkg, echo):
    good = [0, 0, 0, 0.0, None, None, 0, 0.0, None, 0, 0, None]
    for call in _callers(pkg, echo):
        call(*good)
        for at, bad in ((0, object()), (2, None), (3, "x"), (9, 1.5)):
            with pytest.raises((TypeError, C.ArgumentError, AttributeError)):
                call(*(good[:at] + [bad] + good[at + 1:]))
        with pytest.raises(TypeError):
            call(*good[:-1])


def test_signatures_are_the_headers(pkg):
    text = re.sub(r"/\*.*?\*/", "", open(os.path.join(ROOT, "include", "goph_b200.h")).read(), flags=re.S)
    protos = dict(re.findall(r"\bint\s+(goph_[a-z0-9_]+)\s*\(([^)]*)\)", text))
    for name, sig in pkg.runtime._HOT.items():
        kinds = "".join("p" if "*" in a else "n" if "uint64_t" in a else "f" if "float" in a else "i" for a in protos[name].split(","))
        assert sig == kinds, name


def test_the_library_without_the_module(pkg, monkeypatch):
    """Another Python than the build's finds no module of its own and calls through ctypes."""
    rt = pkg.runtime
    if not os.path.exists(rt.LIB_PATH):
        pkg.build.build()
    monkeypatch.setattr(rt.sysconfig, "get_config_var", lambda name: ".cpython-000-nowhere.so")
    assert rt._pycall() is None
    monkeypatch.setattr(rt, "_lib", None)
    L = rt.lib()
    assert isinstance(L.goph_mlx_gemv, C._CFuncPtr)
    assert L.goph_mlx_gemv(None, 0, None, 0, None, None) == 1
    assert L.goph_mlx_gemv(1 << 40, 1 << 40, b"addresses", C.c_uint64(5), C.c_void_p(0), None) == 1   # (nil handle)
