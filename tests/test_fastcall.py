"""The extension that calls the library without ctypes' conversions hands over what ctypes would: every signature of the binding, called
through both into a recorder (no device needed)."""
import ctypes as C

import pytest

from mlx_parallm_b200 import _lib

fast = pytest.importorskip("mlx_parallm_b200._fastcall")
BOUND = sorted(n for n, (res, args) in _lib.SIGNATURES.items() if res is C.c_int and all(a in _lib._LETTERS for a in args))


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


def test_scratch_views_are_kept_and_follow_a_new_allocation():
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
    s.allocate()
    assert s.get("a", torch.float32, 3, 4).data_ptr() == s._bufs[("a", torch.float32)].data_ptr()
