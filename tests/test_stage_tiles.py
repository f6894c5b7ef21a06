"""The nonlinear stage on halo tiles (csrc/mpsw_stage.h), run on the host tile by tile: tendencies
and linearisation point equal the oracle's bit for bit whatever the tile size and the physics, every
entity is owned by one tile, and the tiles stay within the caps of a block."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

import oracle as O
from helpers import setup

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), 'mpas-sw-tl-ad_b200', 'csrc')


@pytest.fixture(scope='module')
def lib(tmp_path_factory):
    gxx = shutil.which('g++')
    if not gxx:
        pytest.skip('no g++')
    out = str(tmp_path_factory.mktemp('stage') / 'libstagecheck.so')
    subprocess.run([gxx, '-O2', '-std=c++17', '-ffp-contract=off', '-shared', '-fPIC', '-I' + CSRC,
                    os.path.join(CSRC, 'mpsw_setup.cpp'), os.path.join(CSRC, 'mpsw_tiles.cpp'),
                    os.path.join(HERE, 'stage_check.cpp'), '-o', out], check=True)
    return ctypes.CDLL(out)


def run(lib, m, K):
    keep = []

    def ptrs(names, dt):
        arrs = [np.ascontiguousarray(np.asarray(getattr(m, n)).T, dtype=dt) for n in names]
        keep.extend(arrs)
        return (ctypes.c_void_p * len(arrs))(*[a.ctypes.data for a in arrs])
    ints = np.array([m.ncells, m.nedges, m.nvertices, m.maxedges, m.maxedges2, K], dtype=np.int32)
    cfg = np.array([m.config_dt, m.config_apvm_upwinding, m.config_h_mom_eddy_visc2, m.config_h_mom_eddy_visc4,
                    float(m.config_bottom_drag), float(m.config_wind_stress)], dtype=np.float64)
    conn = ptrs(['cellsonedge', 'verticesonedge', 'edgesonedge', 'nedgesonedge', 'edgesoncell', 'nedgesoncell',
                 'cellsonvertex', 'edgesonvertex'], np.int32)
    met = ptrs(['weightsonedge', 'kiteareasonvertex', 'dcedge', 'dvedge', 'areacell', 'areatriangle', 'fvertex',
                'h_s', 'u_src', 'xcell', 'ycell', 'zcell', 'xedge', 'yedge', 'zedge', 'xvertex', 'yvertex',
                'zvertex'], np.float64)
    nE, nC, nV = int(m.nedges), int(m.ncells), int(m.nvertices)
    outs = [np.empty(n) for n in (nE, nC) + (nE,) * 6 + (nV, nV, nC)]
    po = (ctypes.c_void_p * 11)(*[a.ctypes.data for a in outs])
    u, h = m.u[0, 0].copy(), m.h[0, 0].copy()
    counts = np.zeros(14, dtype=np.int64)
    err = ctypes.create_string_buffer(512)
    rc = lib.stage_check(ints.ctypes.data_as(ctypes.c_void_p), cfg.ctypes.data_as(ctypes.c_void_p), conn, met,
                         u.ctypes.data_as(ctypes.c_void_p), h.ctypes.data_as(ctypes.c_void_p), po,
                         counts.ctypes.data_as(ctypes.c_void_p), err, 512)
    assert rc == 0, err.value.decode()
    return outs, counts


@pytest.mark.parametrize('phys', [dict(), dict(visc2=1e5, drag=True), dict(visc2=2e5, visc4=1e15, drag=True, wind=True)])
@pytest.mark.parametrize('level,K', [(0, 1), (0, 64), (1, 5), (3, 1), (3, 17), (4, 70)])
def test_stage_equals_the_oracle(lib, level, K, phys):
    o = setup(O.OracleModule(), level, 'seeded', **phys)
    outs, counts = run(lib, o, K)
    o.solve_diagnostics()
    o.compute_tend()
    assert counts[3] == 0 and counts[4] == 0
    names = ['tend_u', 'tend_h', 'u', 'h_edge', 'v', 'gradpvt', 'gradpvn', 'pv_edge', 'vorticity', 'h_vertex', 'ke']
    for n, x in zip(names, outs):
        assert np.array_equal(x, np.asarray(getattr(o, n))[0].ravel()), n


def test_stage_tiles_keep_the_caps(lib):
    o = setup(O.OracleModule(), 5, 'balanced')
    outs, counts = run(lib, o, 1000)
    assert counts[0] >= 148 and counts[2] == 0 and counts[3] == 0
    o.compute_tend()
    assert np.array_equal(outs[0], o.tend_u[0])
