"""The bounds-checked build's checks of the fixed-point solve's pointer loops,
on the CPU: they pass what stays inside and stop what does not."""
import ctypes

import pytest

import fx_host


def bounds(what, n, count, ns, extra):
    changed = ctypes.c_int(-1)
    f = fx_host.lib("fx_bounds.cpp").fxh_bounds
    f.restype = ctypes.c_longlong
    hits = f(what, n, count, ns, extra, ctypes.byref(changed))
    assert changed.value == 0
    return hits


# (loop, order, vectors, length, place of the reflector's vector or of the chunk's element)
@pytest.mark.parametrize("what,n,count,ns,extra", [(0, 8, 8, 7, 7), (0, 8, 8, 3, 0), (1, 8, 8, 7, 0), (1, 8, 0, 9, 0),
                                                  (2, 8, 0, 0, 15), (3, 8, 0, 0, 1)])
def test_inside(what, n, count, ns, extra):
    assert bounds(what, n, count, ns, extra) == 0


@pytest.mark.parametrize("what,n,count,ns,extra", [(0, 8, 9, 7, 0), (0, 8, 8, 7, 8), (1, 8, 9, 7, 0), (1, 8, 8, 8, 0),
                                                  (2, 8, 0, 0, 16), (2, 8, 0, 0, -1), (3, 8, 0, 0, 2)])
def test_outside_is_counted_and_not_taken(what, n, count, ns, extra):
    assert bounds(what, n, count, ns, extra) > 0
