"""A window whose stages are stored in both precisions: one forward sweep serves both, so a sweep in the
second precision launches its own kernels and at most one rounding, gives the results of a window used in that
precision alone, and is linearised about the trajectory that the first sweep integrated even where the
namelist has changed since.  A store that is allocated after a sweep was captured is written as well."""
import numpy as np
import pytest

from helpers import setup
from module_sw_mpas import MpasSwModule

pytestmark = pytest.mark.gpu
torch = pytest.importorskip('torch')


def members(m, B, seed):
    rng = np.random.default_rng(seed)
    return (torch.tensor(rng.standard_normal((int(m.nedges), B)) * 0.1, device='cuda'),
            torch.tensor(rng.standard_normal((int(m.ncells), B)), device='cuda'))


@pytest.mark.parametrize('tiles', ['1', '0'])
@pytest.mark.parametrize('first', [0, 1])
def test_one_forward_serves_both_precisions(monkeypatch, tiles, first):
    from mpsw.torch_api import Engine
    monkeypatch.setenv('MPSW_STAGE_TILES', tiles)
    m = setup(MpasSwModule(), 3, 'seeded', dt=600.0)
    e = Engine(m)
    x, y, other, lib = members(m, 3, 1), members(m, 3, 2), 1 - first, m.handle.lib
    for prec in (0, 1):
        e.window(4).tl(*x, prec)  # tuned, and its buffers allocated
        e.window(4).ad(*y, prec)
    alone = e.window(4).ad(*y, other)
    w = e.window(4)
    w.tl(*x, first)
    n = [lib.mpsw_launch_count()]
    for _ in range(2):
        both = w.ad(*y, other)
        n.append(lib.mpsw_launch_count())
    assert n[1] - n[0] <= n[2] - n[1] + 1
    for a, b in zip(both, alone):
        assert torch.equal(a, b)


@pytest.mark.parametrize('prec', [0, 1])
def test_second_precision_after_a_change_of_viscosity(prec):
    from mpsw.torch_api import Engine
    out = []
    for sweep_first in (True, False):
        m = setup(MpasSwModule(), 3, 'seeded', dt=600.0)
        e = Engine(m)
        x, y = members(m, 2, 1), members(m, 2, 2)
        w = e.window(3)
        w.tl(*x, 1 - prec) if sweep_first else w.final_state()
        m.config_h_mom_eddy_visc2 = 1.0e6
        out.append(w.ad(*y, prec))
    for a, b in zip(*out):
        assert torch.equal(a, b)


def test_store_allocated_after_a_sweep():
    from mpsw.torch_api import FP32, FP64, Engine
    m = setup(MpasSwModule(), 3, 'seeded', dt=600.0)
    e = Engine(m)
    x, y = members(m, 4, 1), members(m, 4, 2)
    want = e.window(4, storage=1).ad(*y, FP64)
    e.window(4, storage=2).tl(*x, FP32)  # (frees the FP64 store)
    w = e.window(4, storage=3)
    w.tl(*x, FP32)
    for a, b in zip(w.ad(*y, FP64), want):
        assert torch.equal(a, b)
