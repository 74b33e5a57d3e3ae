"""The extension module that calls entry points: every kind of argument arrives as the function's own signature says."""
import ctypes
import platform

import pytest

from ultima_b200.kernels import build

P, I, L, U, F = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_ulonglong, ctypes.c_float
needs_module = pytest.mark.skipif(not build.calls_can_be_built(), reason="this host calls entry points through ctypes")


def _bound(types, fn):
    kind = ctypes.CFUNCTYPE(I, *types)
    held = kind(fn)
    return held, build._bind()(ctypes.cast(held, P).value, "".join(build._CODES[t] for t in types))


@needs_module
@pytest.mark.parametrize("n_ints", [0, 1, 5, 6, 7, 33, 48])
@pytest.mark.parametrize("n_floats", [0, 1, 8])
def test_arguments_of_every_kind_keep_their_order_and_values(n_ints, n_floats):
    kinds = [(I, -7), (L, -(1 << 40)), (P, (1 << 47) + 8), (U, (1 << 63) + 5)]
    types, values, got = [], [], []
    for i in range(max(n_ints, n_floats)):                       # integers and floats in turn
        if i < n_ints:
            t, v = kinds[i % 4]
            types.append(t)
            values.append(v + i)
        if i < n_floats:
            types.append(F)
            values.append(i + 0.25)
    held, call = _bound(types, lambda *a: got.append(a) or 41)
    assert call(*values) == 41
    assert [v or 0 for v in got[0]] == [v or 0 for v in values]


@needs_module
def test_none_arrays_numpy_integers_and_what_is_refused():
    import numpy as np
    got = []
    held, call = _bound([P, P, I, F], lambda *a: got.append(a) or 0)
    arr = (ctypes.c_float * 3)(1, 2, 3)
    assert call(None, arr, np.int64(9), 2) == 0
    assert got[0] == (None, ctypes.addressof(arr), 9, 2.0)
    for bad in ((1, 2, 3), (1, 2, 3, 4.0, 5), (1, 2, None, 1.0), (1, 2, 1.5, 1.0), (1, 2, 3, "x")):
        with pytest.raises(TypeError):
            call(*bad)
    with pytest.raises(ValueError):
        build._bind()(ctypes.cast(held, P).value, "F" * 9)


@needs_module
def test_pointers_are_what_ctypes_takes_for_them_and_nothing_else():
    """The same words, and the same refusals, as the foreign call that the module stands in for."""
    import numpy as np
    got = []
    held, call = _bound([P], lambda a: got.append(a) or 0)
    x, arr = ctypes.c_int(5), (ctypes.c_int * 4)(1, 2, 3, 4)
    for value, word in ((P(4096), 4096), (P(None), None), (ctypes.pointer(x), ctypes.addressof(x)), (ctypes.byref(x), ctypes.addressof(x)),
                        (ctypes.cast(arr, ctypes.POINTER(ctypes.c_int)), ctypes.addressof(arr)), (arr, ctypes.addressof(arr)),
                        (1 << 47, 1 << 47)):
        assert call(value) == 0 and got.pop() == word
        assert held(value) == 0 and got.pop() == word
    for refused in (np.zeros(4, np.float32), bytearray(8), memoryview(b"abcd"), x, 1.5, [1]):
        for f in (call, held):
            with pytest.raises((TypeError, ctypes.ArgumentError)):
                f(refused)
    assert got == []


@pytest.fixture
def other_host(monkeypatch):
    """The loader as on a host that has not been asked yet, put back afterwards."""
    build.calls_can_be_built.cache_clear()
    monkeypatch.setattr(build, "_calls", None)
    yield monkeypatch
    monkeypatch.undo()
    build.calls_can_be_built.cache_clear()


@pytest.mark.parametrize("what", ["an Arm host", "another system", "Python 3.11", "another Python", "no headers"])
def test_a_host_that_cannot_build_the_module_keeps_ctypes(what, other_host, tmp_path):
    from ultima_b200.kernels import catalog
    if what == "an Arm host":
        other_host.setattr(platform, "machine", lambda: "aarch64")
    elif what == "another system":
        other_host.setattr(build.sys, "platform", "win32")
    elif what == "Python 3.11":
        other_host.setattr(build.sys, "version_info", (3, 11, 9, "final", 0))
    elif what == "another Python":
        other_host.setattr(build.sys, "implementation", type("I", (), {"name": "pypy"}))
    else:
        other_host.setattr(build, "_python_include", lambda: str(tmp_path))
    asked = []
    other_host.setattr(build, "ensure_built", lambda targets: asked.extend(targets) or {})
    lib = ctypes.CDLL(None)
    assert not build.calls_can_be_built() and build.native(lib) is lib
    assert (build.CALLS, ()) not in catalog.all_targets()
    build.prebuild([])
    assert asked == []


def test_a_module_that_fails_to_build_is_an_error_every_time(other_host):
    def fails(targets):
        raise build.BuildError("no compiler")
    other_host.setattr(build, "calls_can_be_built", lambda: True)
    other_host.setattr(build, "ensure_built", fails)
    for _ in range(2):
        with pytest.raises(build.BuildError):
            build.native(ctypes.CDLL(None))
