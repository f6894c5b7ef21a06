"""Which calls take the stages on halo tiles: with tiles a forward, a tangent linear and an adjoint launch
fewer kernels than with MPSW_STAGE_TILES=0, in the cases that the dispatch sends there and in no others, and
FP64 results are the passes' bit for bit on either route."""
import numpy as np
import pytest

from helpers import setup
from module_sw_mpas import MpasSwModule

pytestmark = pytest.mark.gpu
torch = pytest.importorskip('torch')

VISC2, FULL = dict(visc2=1e5, drag=True), dict(visc2=1e5, visc4=5e14, drag=True, wind=True)


def members(e, B, seed):
    rng = np.random.default_rng(seed)
    return (torch.tensor(rng.standard_normal((e.nE, B)) * 0.1, device='cuda'), torch.tensor(rng.standard_normal((e.nC, B)), device='cuda'))


def launches(lib, f):
    f()  # tuned, allocated, captured
    n = lib.mpsw_launch_count()
    out = f()
    return lib.mpsw_launch_count() - n, out


# level, precision, members, physics; whether the tangent linear and the adjoint run on tiles, and the forward
# that a sweep recomputes
@pytest.mark.parametrize('level,prec,B,phys,tl,ad,between', [
    (3, 0, 1, {}, True, True, True), (3, 0, 2, {}, True, True, True), (3, 0, 3, {}, False, False, True),
    (3, 0, 1, VISC2, True, False, True), (3, 0, 2, FULL, True, False, True), (3, 1, 5, FULL, False, False, True),
    (6, 0, 1, {}, True, True, True), (6, 0, 2, {}, False, False, True), (6, 0, 1, FULL, False, False, True),
    (6, 0, 2, FULL, False, False, False), (6, 1, 32, FULL, False, False, True), (6, 1, 40, FULL, False, False, False)])
def test_routes(monkeypatch, level, prec, B, phys, tl, ad, between):
    from mpsw.torch_api import Engine
    res = []
    for tiles in ('1', '0'):
        monkeypatch.setenv('MPSW_STAGE_TILES', tiles)
        m = setup(MpasSwModule(), level, 'seeded', dt=75.0 * 2 ** (7 - level), **phys)
        e, lib = Engine(m), m.handle.lib
        x, y = members(e, B, 1), members(e, B, 2)
        stored = e.window(2)
        stored.tl(*x, prec)
        n = [launches(lib, lambda: m.handle.call('mpsw_forward', 0, 1))[0]]
        r = []
        for f in (lambda: stored.tl(*x, prec), lambda: stored.ad(*y, prec)):
            k, out = launches(lib, f)
            n.append(k)
            r += out
        bare = e.window(1, storage=0)  # (one step: no replay of the forward)
        for f in (lambda: bare.tl(*x, prec), lambda: bare.ad(*y, prec)):
            k, out = launches(lib, f)
            n.append(k)
            r += out
        res.append((n, r))
    (nt, rt), (npass, rp) = res
    assert nt[0] < npass[0]
    assert (nt[1] < npass[1], nt[2] < npass[2]) == (tl, ad)
    assert (nt[3] < npass[3], nt[4] < npass[4]) == (between or tl, between or ad)
    for a, b in zip(rt, rp):
        if prec == 0:
            assert torch.equal(a, b)
        else:  # (the members' kernels are the same; the tuner may give them another width: one rounding)
            assert float((a - b).norm()) <= 1e-6 * float(b.norm())
