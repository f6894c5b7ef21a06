"""Launch choices are kept apart for the kernels that the sweeps run: physics that sends a sweep to the
general passes tunes those, and a cache file written with row passes gives no choices to a mesh without."""
import ctypes

import numpy as np
import pytest

from helpers import setup
from module_sw_mpas import MpasSwModule

pytestmark = pytest.mark.gpu
torch = pytest.importorskip('torch')

AD_EDGE, AD_VERTEX, TL_VERTEX = 4, 6, 0  # kernels of mpsw_window_tuning's table


def sweep(e, B, prec):
    rng = np.random.default_rng(0)
    x = (torch.tensor(rng.standard_normal((e.nE, B)), device='cuda'), torch.tensor(rng.standard_normal((e.nC, B)), device='cuda'))
    w = e.window(2)
    return w.ad(*w.tl(*x, prec), prec)


def choice(e, B, prec, kernel):
    v = (ctypes.c_int * 16)()
    e.h.call('mpsw_window_tuning', prec, B, v)
    return v[2 * kernel], v[2 * kernel + 1]


@pytest.mark.parametrize('prec,B,kernel', [(1, 16, AD_VERTEX), (0, 1, AD_EDGE)])
def test_viscosity_tunes_the_general_passes(prec, B, kernel):
    from mpsw.torch_api import Engine
    m = setup(MpasSwModule(), 3, 'seeded', dt=600.0)
    e = Engine(m)
    sweep(e, B, prec)
    assert choice(e, B, prec, kernel) == (0, 0)
    m.config_h_mom_eddy_visc2 = 1.0e5
    a = sweep(e, B, prec)
    assert all(choice(e, B, prec, kernel))
    m.config_h_mom_eddy_visc2 = 0.0
    assert choice(e, B, prec, kernel) == (0, 0)
    fresh = Engine(setup(MpasSwModule(), 3, 'seeded', dt=600.0, visc2=1.0e5))
    for x, y in zip(a, sweep(fresh, B, prec)):
        assert float((x - y).norm()) <= (1e-6 if prec else 0.0) * float(y.norm())


def test_cache_file_is_for_the_kernels_that_run(tmp_path, monkeypatch):
    from mpsw.torch_api import Engine
    monkeypatch.setenv('MPSW_TUNE_CACHE', str(tmp_path / 'tune.txt'))
    for rows in ('1', '0', '1'):
        monkeypatch.setenv('MPSW_ROWS', rows)
        e = Engine(setup(MpasSwModule(), 3, 'seeded', dt=600.0))
        sweep(e, 16, 1)
        assert all(choice(e, 16, 1, TL_VERTEX)) == (rows == '0')
    assert len((tmp_path / 'tune.txt').read_text().split()) == 2 * 17
