"""Values set on a variable that a routine has since written on the device: contents that were exchanged
before are taken over again, through the ABI and as attributes of the module, while an array that nobody
touched leaves a value that was written through the handle alone."""
import ctypes

import numpy as np
import pytest

from helpers import setup
from module_sw_mpas import MpasSwModule

pytestmark = pytest.mark.gpu


def update(h, name, x):
    h.call('mpsw_update_var', name, x.ctypes.data_as(ctypes.c_void_p), x.size)


def get(h, name, like):
    x = np.empty_like(like)
    h.call('mpsw_get_var', name, x.ctypes.data_as(ctypes.c_void_p), x.size)
    return x


def test_update_resets_what_a_routine_wrote():
    m = setup(MpasSwModule(), 2, 'tc5')
    h = m.handle
    u0, h0 = m.u.copy(order='F'), m.h.copy(order='F')
    for _ in range(2):
        update(h, b'u', u0)
        update(h, b'h', h0)
        h.call('mpsw_sw_rk4', 1)
        h.call('mpsw_edit_var', b'u', u0.ctypes.data_as(ctypes.c_void_p), u0.size)  # unedited: the result stands
    first = setup(MpasSwModule(), 2, 'tc5')
    first.sw_rk4()
    assert np.array_equal(get(h, b'u', u0), first.u) and np.array_equal(get(h, b'h', h0), first.h)


def test_assignment_after_a_routine():
    m = setup(MpasSwModule(), 2, 'tc5', ad=True)
    rng = np.random.default_rng(0)
    seed, ua = rng.standard_normal(m.tend_u_ad.shape), rng.standard_normal(m.u_ad.shape)
    out = []
    for _ in range(2):
        m.tend_u_ad = seed  # read lazily, and zeroed by the routine
        m.u_ad = ua
        m.h_ad = np.zeros(m.h_ad.shape)
        m.sw_rk4_adj()
        out.append((m.u_ad.copy(), m.h_ad.copy()))
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    assert not m.tend_u_ad.any()


def test_unstable_step_is_taken_back():
    m = setup(MpasSwModule(), 2, 'tc5', dt=600.0)
    u0, h0 = m.u.copy(order='F'), m.h.copy(order='F')
    m.config_dt = 1e200
    with pytest.raises(RuntimeError):
        for _ in range(5):
            m.sw_rk4()
    m.config_dt = 600.0
    m.u, m.h = u0, h0
    m.sw_rk4()
    ref = setup(MpasSwModule(), 2, 'tc5', dt=600.0)
    ref.sw_rk4()
    assert np.array_equal(m.u, ref.u) and np.array_equal(m.h, ref.h)


def test_untouched_array_leaves_the_device_value():
    m, ref = setup(MpasSwModule(), 2, 'tc5'), setup(MpasSwModule(), 2, 'tc5')
    m.handle.call('mpsw_sw_rk4', 2)
    m.sw_rk4()
    for _ in range(3):
        ref.sw_rk4()
    assert np.array_equal(m.u, ref.u) and np.array_equal(m.h, ref.h)
    u = m.u  # edited in place, through a reference held over a call
    m.sw_rk4()
    u[0, 0, 5] += 1.0
    want = u.copy()
    m.sync()
    assert np.array_equal(get(m.handle, b'u', u), want)
