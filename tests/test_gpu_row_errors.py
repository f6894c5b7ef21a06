"""Rounding errors of the FP32 member-row passes (csrc/mpsw_rows.cuh): their results are as close to FP64
members' as those of the general passes (MPSW_ROWS=0 when the mesh is built), for independent
perturbations and for smooth ones, where differences of neighbouring rows cancel.  One stage of the row
passes in emulated FP32 has 0.5 to 1.02 times the error of the general passes (levels 3 to 5, u and h, both
directions); the stages of a window add theirs alike, and the members' mean leaves a few per cent of
scatter: 1.1."""
import numpy as np
import pytest

from helpers import mesh, setup
from module_sw_mpas import MpasSwModule
from mpsw import ic

pytestmark = pytest.mark.gpu
torch = pytest.importorskip('torch')

MARGIN = 1.1


def perturbation(level, kind, B, seed):
    m = ic.scale_mesh(mesh(level))
    rng = np.random.default_rng(seed)
    if kind == 'white':
        return 0.1 * rng.standard_normal((m['nEdges'], B)), rng.standard_normal((m['nCells'], B))
    flows = [ic.balanced_flow(m, 10 * seed + s) for s in range(6)]
    c = rng.standard_normal((6, B))
    u = np.stack([f['u'] for f in flows], 1) @ c
    h = np.stack([f['h'] - f['h'].mean() for f in flows], 1) @ c
    if kind == 'height':
        u = u * 0.0
    return u / 400.0, h / 400.0


def error(a, ref):
    return [float(((x - r).norm(dim=0) / r.norm(dim=0)).mean()) for x, r in zip(a, ref)]


@pytest.mark.parametrize('cfg', [dict(), dict(visc2=1e5, drag=True), dict(visc2=1e5, visc4=5e14, drag=True, wind=True)])
@pytest.mark.parametrize('level,B', [(4, 24), (5, 64), (6, 16)])
def test_row_errors_are_the_general_passes(monkeypatch, level, B, cfg):
    from mpsw.torch_api import FP32, FP64, Engine
    engines = []
    for rows in ('1', '0'):
        monkeypatch.setenv('MPSW_ROWS', rows)
        engines.append(Engine(setup(MpasSwModule(), level, 'seeded', dt=75.0 * 2 ** (7 - level), **cfg)))
    for kind in ('white', 'smooth', 'height'):
        x, y = (tuple(torch.tensor(a, device='cuda') for a in perturbation(level, kind, B, s)) for s in (1, 2))

        def sweeps(e, prec):
            w = e.window(4, ckpt_every=2)
            return w.tl(*x, prec), w.ad(*y, prec)
        ref, rows, general = sweeps(engines[1], FP64), sweeps(engines[0], FP32), sweeps(engines[1], FP32)
        for i, what in enumerate(('tl', 'ad')):
            for er, eg in zip(error(rows[i], ref[i]), error(general[i], ref[i])):
                assert er <= MARGIN * eg, (kind, what, er, eg)
