"""The extension module that calls entry points: every kind of argument arrives as the function's own signature says."""
import ctypes

import pytest

from ultima_b200.kernels import build

P, I, L, U, F = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_ulonglong, ctypes.c_float
pytestmark = pytest.mark.skipif(not build.calls_can_be_built(), reason="Python's headers are not here")


def _bound(types, fn):
    kind = ctypes.CFUNCTYPE(I, *types)
    held = kind(fn)
    return held, build._bind()(ctypes.cast(held, P).value, "".join(build._CODES[t] for t in types))


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
