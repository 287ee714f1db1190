"""The extension that calls the library without ctypes' conversions hands over what ctypes would: every signature of the binding, called
through both into a recorder (no device needed)."""
import ctypes as C
import os
import platform
import shutil
import subprocess
import sys
import sysconfig

import pytest

from mlx_parallm_b200 import _lib

fast = _lib._fastcall
needs_fast = pytest.mark.skipif(fast is None, reason="the extension is not built for this interpreter")
CSRC = os.path.join(os.path.dirname(_lib.__file__), "csrc")
BUILDABLE = os.path.exists(os.path.join(sysconfig.get_paths()["include"], "Python.h")) and platform.machine() == "x86_64" and sys.platform == "linux"
BOUND = sorted(n for n, (res, args) in _lib.SIGNATURES.items() if res is C.c_int and all(a in _lib._LETTERS for a in args))


@pytest.mark.skipif(not BUILDABLE or not os.path.exists(os.path.join(os.path.dirname(_lib.__file__), "libb200parallm.so")), reason="nothing built, or no headers")
def test_a_built_tree_has_the_extension_of_this_interpreter():
    assert fast is not None and fast.__file__.endswith(sysconfig.get_config_var("EXT_SUFFIX"))


@pytest.mark.skipif(not BUILDABLE, reason="no Python headers, or another platform")
def test_the_build_reports_what_it_does_not_build(tmp_path):
    """A compile error fails the build, a missing header is said, and the file carries the interpreter's suffix (another one does not load it)."""
    os.mkdir(tmp_path / "csrc")
    for f in ("Makefile", "fastcall.c"):
        shutil.copy(os.path.join(CSRC, f), tmp_path / "csrc" / f)
    make = lambda *a: subprocess.run(["make", "-C", str(tmp_path / "csrc"), "fast", *a], capture_output=True, text=True)        # noqa: E731
    skipped = make("PYTHON=/nonexistent/python")
    assert skipped.returncode == 0 and "not built" in skipped.stdout
    assert make("PYTHON=" + sys.executable).returncode == 0
    assert [f for f in os.listdir(tmp_path) if f.startswith("_fastcall")] == ["_fastcall" + sysconfig.get_config_var("EXT_SUFFIX")]
    with open(tmp_path / "csrc" / "fastcall.c", "a") as f:
        f.write("int broken(void) { return undeclared; }\n")
    os.utime(tmp_path / "csrc" / "fastcall.c", (2 ** 31, 2 ** 31))
    assert make("PYTHON=" + sys.executable).returncode != 0


@needs_fast
@pytest.mark.parametrize("name", BOUND)
def test_arguments_arrive(name):
    args = _lib.SIGNATURES[name][1]
    seen = []
    proto = C.CFUNCTYPE(C.c_int, *args)
    target = proto(lambda *a: (seen.append(a), -3)[1])
    f = fast.bind(C.cast(target, C.c_void_p).value, "".join(_lib._LETTERS[a] for a in args), target)
    values = []
    for i, a in enumerate(args):
        if a is C.c_float:
            values.append(0.5 + i)
        elif a is C.c_void_p:
            values.append(None if i % 3 == 1 else 0x7f0000001000 + 16 * i)
        elif a is C.c_int:
            values.append(-7 - i if i % 2 else 2 ** 31 - 1 - i)
        else:
            values.append(2 ** 40 + i if a in (C.c_uint64, C.c_size_t) or i % 2 else -(2 ** 40) - i)
    assert f(*values) == -3 and target(*values) == -3
    assert seen[0] == seen[1] and len(seen[0]) == len(args)


@needs_fast
def test_other_arguments_go_through_ctypes():
    seen = []
    target = C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_int, C.c_float)(lambda *a: (seen.append(a), 0)[1])
    f = fast.bind(C.cast(target, C.c_void_p).value, "pif", target)
    assert f(C.c_void_p(64), True, 2) == 0 and seen == [(64, 1, 2.0)]      # a ctypes object, a truth value, an integer for a float
    for bad in ((object(), 1, 1.0), (1, 1.5, 1.0), (1, 1)):
        with pytest.raises((C.ArgumentError, TypeError)):
            f(*bad)
    with pytest.raises(ValueError):
        fast.bind(1, "pq", target)
    with pytest.raises(ValueError):
        fast.bind(1, "f" * 9, target)


def test_error_codes_and_messages():
    L = _lib.lib()
    assert L.b200p_qmm_set_path(7) == -1 and "path" in _lib.last_error()
    with pytest.raises(_lib.B200PError):
        _lib.check(L.b200p_gemm(None, None, None, *[1] * 10, 0, 0, 0.0, 0.0, None), "b200p_gemm")


def test_scratch_views_are_kept_and_follow_a_new_allocation(monkeypatch):
    import torch
    from mlx_parallm_b200.models._sequence import Scratch
    s = Scratch(torch.device("cpu"), 700)
    s.reserve("a", torch.float32, 4)
    s.allocate()
    v = s.get("a", torch.float32, 3, 4)
    assert v.shape == (3, 4) and s.get("a", torch.float32, 3, 4) is v and s.get("a", torch.float32, 6, 2).data_ptr() == v.data_ptr()
    for m in range(1, 700):
        assert s.get("a", torch.float32, m, 4).shape == (m, 4)
    assert len(s._views) <= 512
    del v
    s.reserve("b", torch.float32, 4)
    make, held = torch.empty, []
    monkeypatch.setattr(torch, "empty", lambda *args, **kw: (held.append(len(s._views)), make(*args, **kw))[1])
    s.allocate()
    assert held == [0, 0]                                    # no view keeps a buffer that is being replaced
    assert s.get("a", torch.float32, 3, 4).data_ptr() == s._bufs[("a", torch.float32)].data_ptr()
