"""Tables of the FP64 adjoint stage's tiles (csrc/mpsw_stage.h): every neighbour that a phase reads lies in
the layer that the phase before has formed, every cell and edge has one owner, the layers stay within a
block's caps and the blobs are 16-byte aligned, whatever the tile size.  (Their results are compared with the
passes' bit for bit on the GPU, test_gpu_stage_tiles.py.)"""
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
    out = str(tmp_path_factory.mktemp('stage_ad') / 'libstageadcheck.so')
    subprocess.run([gxx, '-O2', '-std=c++17', '-shared', '-fPIC', '-I' + CSRC, os.path.join(CSRC, 'mpsw_setup.cpp'),
                    os.path.join(CSRC, 'mpsw_tiles.cpp'), os.path.join(HERE, 'stage_ad_check.cpp'), '-o', out], check=True)
    return ctypes.CDLL(out)


@pytest.mark.parametrize('level,K', [(0, 1), (0, 64), (1, 5), (3, 1), (3, 18), (4, 40), (5, 96)])
def test_tables(lib, level, K):
    m = setup(O.OracleModule(), level, 'seeded')
    keep = []

    def ptrs(names, dt):
        arrs = [np.ascontiguousarray(np.asarray(getattr(m, n)).T, dtype=dt) for n in names]
        keep.extend(arrs)
        return (ctypes.c_void_p * len(arrs))(*[a.ctypes.data for a in arrs])
    ints = np.array([m.ncells, m.nedges, m.nvertices, m.maxedges, m.maxedges2, K], dtype=np.int32)
    conn = ptrs(['cellsonedge', 'verticesonedge', 'edgesonedge', 'nedgesonedge', 'edgesoncell', 'nedgesoncell',
                 'cellsonvertex', 'edgesonvertex'], np.int32)
    met = ptrs(['weightsonedge', 'kiteareasonvertex', 'dcedge', 'dvedge', 'areacell', 'areatriangle', 'fvertex',
                'h_s', 'u_src', 'xcell', 'ycell', 'zcell', 'xedge', 'yedge', 'zedge', 'xvertex', 'yvertex',
                'zvertex'], np.float64)
    counts, err = np.zeros(5, dtype=np.int64), ctypes.create_string_buffer(512)
    rc = lib.stage_ad_check(ints.ctypes.data_as(ctypes.c_void_p), conn, met, counts.ctypes.data_as(ctypes.c_void_p),
                            err, 512)
    assert rc == 0, err.value.decode()
    assert counts[0] >= -(-int(m.ncells) // K)
    assert not counts[1:].any(), counts
