"""mpsw_var_changed on the host side: tells edited contents from those last exchanged, takes nothing over,
and refuses what mpsw_set_var refuses."""
import ctypes

import numpy as np

from test_transfers import get, handle


def test_tells_edits_and_takes_nothing_over():
    h = handle(30)
    x = np.arange(60.0)
    p = x.ctypes.data_as(ctypes.c_void_p)
    c = ctypes.c_int(-1)

    def changed():
        h.call('mpsw_var_changed', b'u', p, 60, ctypes.byref(c))
        return c.value
    assert changed() == 1  # against the zeros of the allocation
    assert not get(h, ['u'], [60])[0].any()
    h.call('mpsw_set_var', b'u', p, 60)
    assert changed() == 0
    x[59] = np.nan
    assert changed() == 1
    h.call('mpsw_update_var', b'u', p, 60)
    assert changed() == 0 and np.isnan(get(h, ['u'], [60])[0][59])
    for args in ((b'u', p, 59), (b'nothing', p, 60), (b'u', None, 60)):
        assert h.lib.mpsw_var_changed(h.ptr, *args, ctypes.byref(c)) != 0
    assert h.lib.mpsw_var_changed(h.ptr, b'u', p, 60, None) != 0
    h.close()
