"""mpsw_edit_var on the host side: takes edited contents over, and refuses what mpsw_set_var refuses."""
import ctypes

import numpy as np

from test_transfers import get, handle


def test_takes_edits_over():
    h = handle(30)
    x = np.arange(60.0)
    p = x.ctypes.data_as(ctypes.c_void_p)
    h.call('mpsw_edit_var', b'u', p, 60)  # against the zeros of the allocation
    assert np.array_equal(get(h, ['u'], [60])[0], x)
    h.call('mpsw_edit_var', b'u', p, 60)
    x[59] = np.nan
    h.call('mpsw_edit_var', b'u', p, 60)
    assert np.array_equal(get(h, ['u'], [60])[0], x, equal_nan=True)
    for args in ((b'u', p, 59), (b'nothing', p, 60), (b'u', None, 60)):
        assert h.lib.mpsw_edit_var(h.ptr, *args) != 0
    h.close()
