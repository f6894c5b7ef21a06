"""The member-row passes' tables and coefficients (csrc/mpsw_rows.h), run on the host in FP64: a
tangent-linear and an adjoint stage about a random linearisation point equal the same stages formed
through the intermediate fields, the adjoint is the transpose, and a mesh whose lists do not fit the
tables is turned down (its members then take the general passes)."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from helpers import mesh
from mpsw import ic

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), 'mpas-sw-tl-ad_b200', 'csrc')


@pytest.fixture(scope='module')
def lib(tmp_path_factory):
    gxx = shutil.which('g++')
    if not gxx:
        pytest.skip('no g++')
    out = str(tmp_path_factory.mktemp('rows') / 'librowcheck.so')
    subprocess.run([gxx, '-O2', '-std=c++17', '-shared', '-fPIC', '-I' + CSRC, os.path.join(CSRC, 'mpsw_setup.cpp'),
                    os.path.join(CSRC, 'mpsw_rows.cpp'), os.path.join(HERE, 'row_check.cpp'), '-o', out], check=True)
    return ctypes.CDLL(out)


def run(lib, m, seed):
    keep = []

    def ptrs(names, dt):
        arrs = [np.ascontiguousarray(m[n], dtype=dt) for n in names]
        keep.extend(arrs)
        return (ctypes.c_void_p * len(arrs))(*[a.ctypes.data for a in arrs])
    ints = np.array([m['nCells'], m['nEdges'], m['nVertices'], m['maxEdges'], m['maxEdges2'], seed], dtype=np.int32)
    conn = ptrs(['cellsOnEdge', 'verticesOnEdge', 'edgesOnEdge', 'nEdgesOnEdge', 'edgesOnCell', 'nEdgesOnCell',
                 'cellsOnVertex', 'edgesOnVertex'], np.int32)
    met = ptrs(['weightsOnEdge', 'kiteAreasOnVertex', 'dcEdge', 'dvEdge', 'areaCell', 'areaTriangle', 'xCell', 'yCell',
                'zCell', 'xEdge', 'yEdge', 'zEdge', 'xVertex', 'yVertex', 'zVertex'], np.float64)
    out = np.zeros(7)
    err = ctypes.create_string_buffer(512)
    rc = lib.row_check(ints.ctypes.data_as(ctypes.c_void_p), conn, met, out.ctypes.data_as(ctypes.c_void_p), err, 512)
    return rc, err.value.decode(), out


@pytest.mark.parametrize('level', [0, 1, 3, 5])
def test_row_passes_equal_the_general_ones(lib, level):
    rc, err, out = run(lib, ic.scale_mesh(mesh(level)), level)
    assert rc == 0, err
    # tend_u', tend_h', u_ad, h_ad, delsq_u': the same sums in another order; then two dot products
    assert out[:5].max() < 1e-12, out
    assert out[5:].max() < 1e-10, out


def test_other_lists_are_turned_down(lib):
    m = ic.scale_mesh(mesh(2))
    for change in ('short', 'twice'):
        c = dict(m)
        eoe, n = m['edgesOnEdge'].copy(), m['nEdgesOnEdge'].copy()
        if change == 'short':
            n[7] -= 1  # an edge's list without its last entry
        else:
            eoe[7, 1] = eoe[7, 0]
        c['edgesOnEdge'], c['nEdgesOnEdge'] = eoe, n
        rc, err, _ = run(lib, c, 0)
        assert rc == 1 and 'edgesOnEdge' in err
