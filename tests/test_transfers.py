"""Host side of the variable exchange (mpsw_update_var, mpsw_get_vars): content that did not change is
recognised whatever its size (arrays above a few MB are compared and copied in parts), any single
changed value is taken over, and the module reads back what was set."""
import ctypes

import numpy as np
import pytest

from mpsw._lib import Handle


def handle(nE):
    h = Handle()
    for k, v in (('ncells', nE // 3), ('nedges', nE), ('nvertices', 2 * (nE // 3)), ('maxedges', 6), ('maxedges2', 12),
                 ('vertexdegree', 3), ('ntracers', 1), ('nvertlevels', 1)):
        h.check(h.lib.mpsw_set_scalar(h.ptr, k.encode(), float(v)), k)
    h.call('mpsw_var_allocation')
    return h


def get(h, names, sizes):
    n = len(names)
    out = [np.full(s, np.nan) for s in sizes]
    h.call('mpsw_get_vars', n, (ctypes.c_char_p * n)(*[x.encode() for x in names]),
           (ctypes.c_void_p * n)(*[a.ctypes.data for a in out]), (ctypes.c_longlong * n)(*sizes))
    return out


@pytest.mark.parametrize('nE', [30, 131072 + 3, 600001])  # one copy; at the split; four parts with a ragged end
def test_update_takes_every_change(nE):
    h = handle(nE)
    rng = np.random.default_rng(0)
    u, hh = rng.standard_normal(2 * nE), rng.standard_normal(2 * (nE // 3))
    for name, x in (('u', u), ('h', hh)):
        h.call('mpsw_update_var', name.encode(), x.ctypes.data_as(ctypes.c_void_p), x.size)
    for i in (0, nE // 2, nE, 2 * nE - 1):
        u[i] += 1.0
        h.call('mpsw_update_var', b'u', u.ctypes.data_as(ctypes.c_void_p), u.size)
        gu, gh = get(h, ['u', 'h'], [u.size, hh.size])
        assert np.array_equal(gu, u) and np.array_equal(gh, hh)
    u[3] = np.nan
    h.call('mpsw_update_var', b'u', u.ctypes.data_as(ctypes.c_void_p), u.size)
    h.call('mpsw_update_var', b'u', u.ctypes.data_as(ctypes.c_void_p), u.size)
    assert np.isnan(get(h, ['u'], [u.size])[0][3])
    h.close()


def test_bad_arguments_are_refused():
    h = handle(30)
    x = np.zeros(60)
    p = x.ctypes.data_as(ctypes.c_void_p)
    assert h.lib.mpsw_update_var(h.ptr, b'u', p, 59) != 0
    assert h.lib.mpsw_update_var(h.ptr, b'nothing', p, 60) != 0
    assert h.lib.mpsw_update_var(h.ptr, b'u', None, 60) != 0
    with pytest.raises(RuntimeError):
        get(h, ['u', 'h'], [60, 5])
    h.close()
