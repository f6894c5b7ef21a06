"""The stages on halo tiles (csrc/mpsw_stage.cuh) against the grid-wide passes (MPSW_STAGE_TILES=0 when
the mesh is built).  FP64 values are combined in the same order entity by entity, so the tiles' results are
the passes' bit for bit; FP32 stages round some tens of terms differently (1e-5 over these windows)."""
import numpy as np
import pytest

from helpers import setup
from module_sw_mpas import MpasSwModule

pytestmark = pytest.mark.gpu
torch = pytest.importorskip('torch')

CFGS = [dict(), dict(visc2=1e5, drag=True), dict(visc2=1e5, visc4=5e14, drag=True, wind=True), dict(wind=True)]
TOL_FP32 = 1e-5


def module(monkeypatch, tiles, level, **cfg):
    monkeypatch.setenv('MPSW_STAGE_TILES', tiles)
    return setup(MpasSwModule(), level, 'seeded', tl=True, ad=True, dt=300.0, **cfg)


def members(m, B, seed):
    rng = np.random.default_rng(seed)
    return (torch.tensor(rng.standard_normal((int(m.nedges), B)) * 0.1, device='cuda'),
            torch.tensor(rng.standard_normal((int(m.ncells), B)), device='cuda'))


@pytest.mark.parametrize('cfg', CFGS)
@pytest.mark.parametrize('level,B', [(1, 1), (3, 2), (4, 1), (5, 2), (6, 1)])
def test_window_matches_passes(monkeypatch, level, B, cfg):
    from mpsw.torch_api import FP32, FP64, Engine
    out = []
    for tiles in ('1', '0'):
        e = Engine(module(monkeypatch, tiles, level, **cfg))
        x, y = members(e.module, B, 1), members(e.module, B, 2)
        r = []
        for storage in (-1, 0):  # stored and recomputed linearisation points
            w = e.window(3, ckpt_every=2, storage=storage)
            r += w.tl(*x, FP64) + w.ad(*y, FP64)
        w = e.window(3, ckpt_every=2)
        out.append((r, w.tl(*x, FP32) + w.ad(*y, FP32)))
    for a, b in zip(out[0][0], out[1][0]):
        assert torch.equal(a, b)
    for a, b in zip(out[0][1], out[1][1]):
        assert float((a - b).norm()) <= TOL_FP32 * float(b.norm())


@pytest.mark.parametrize('cfg', CFGS)
@pytest.mark.parametrize('level', [1, 3, 5])
def test_steps_match_passes(monkeypatch, level, cfg):
    names = ['u', 'h', 'u_tl', 'h_tl', 'tend_u_tl', 'tend_h_tl', 'u_ad', 'h_ad']
    out = []
    for tiles in ('1', '0'):
        m = module(monkeypatch, tiles, level, **cfg)
        x, y = members(m, 1, 3), members(m, 1, 4)
        m.u_tl[0, 0], m.h_tl[0, 0] = (v[:, 0].cpu().numpy() for v in x)
        for _ in range(2):
            m.sw_rk4_tlm()
        m.u_ad[0, 0], m.h_ad[0, 0] = (v[:, 0].cpu().numpy() for v in y)
        m.sw_rk4_adj()
        out.append([np.array(getattr(m, n)) for n in names])
    for n, a, b in zip(names, *out):
        assert np.array_equal(a, b), n
