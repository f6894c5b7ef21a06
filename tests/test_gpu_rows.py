"""The member-row passes of FP32 members (csrc/mpsw_rows.cuh) against the general passes (MPSW_ROWS=0
when the mesh is built) and the FP64 window: the same sums with folded coefficients, so FP32 roundings
of some tens of terms a stage apart (1e-5 over these windows), and within the FP32-stencil bar of
1e-4 of FP64.  Member counts cover a thread's full vectors, a padded count and several tiles a
block; stored and recomputed linearisation points give the same numbers."""
import numpy as np
import pytest

from helpers import setup
from module_sw_mpas import MpasSwModule

pytestmark = pytest.mark.gpu
torch = pytest.importorskip('torch')

TOL_GENERAL, TOL_FP64 = 1e-5, 1e-4


def engine(monkeypatch, rows, level, **cfg):
    from mpsw.torch_api import Engine
    monkeypatch.setenv('MPSW_ROWS', rows)
    m = setup(MpasSwModule(), level, 'seeded', dt=300.0, **cfg)
    return m, Engine(m)


def members(m, B, seed):
    rng = np.random.default_rng(seed)
    return (torch.tensor(rng.standard_normal((int(m.nedges), B)) * 0.1, device='cuda'),
            torch.tensor(rng.standard_normal((int(m.ncells), B)), device='cuda'))


def sweep(e, x, y, prec, storage=-1):
    w = e.window(5, ckpt_every=2, storage=storage)
    return w.tl(*x, prec) + w.ad(*y, prec)


def relmax(a, b):
    num = torch.sqrt(sum(((p - q) ** 2).sum(0) for p, q in zip(a, b)))
    den = torch.sqrt(sum((q ** 2).sum(0) for q in b))
    return float((num / den).max())


@pytest.mark.parametrize('cfg', [dict(), dict(visc2=1e5, drag=True), dict(visc2=1e5, visc4=5e14, drag=True, wind=True),
                                 dict(wind=True)])
@pytest.mark.parametrize('level,B', [(1, 24), (3, 29), (4, 64), (5, 72)])
def test_rows_match_general_passes(monkeypatch, level, B, cfg):
    from mpsw.torch_api import FP32, FP64
    mr, er = engine(monkeypatch, '1', level, **cfg)
    mg, eg = engine(monkeypatch, '0', level, **cfg)
    x, y = members(mr, B, 1), members(mr, B, 2)
    rows, general, ref = sweep(er, x, y, FP32), sweep(eg, x, y, FP32), sweep(eg, x, y, FP64)
    assert not all(torch.equal(a, b) for a, b in zip(rows, general))  # the row passes did run
    for k in (0, 2):
        assert relmax(rows[k:k + 2], general[k:k + 2]) < TOL_GENERAL
        assert relmax(rows[k:k + 2], ref[k:k + 2]) < TOL_FP64
    for a, b in zip(rows, sweep(er, x, y, FP32, storage=0)):
        assert torch.equal(a, b)
