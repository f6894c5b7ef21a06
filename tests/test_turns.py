"""Pieces of host work over threads (csrc/mpsw_parts.h): each runs once, also where memory runs out while the
threads are started, and the exception of a piece reaches the caller after all have ended."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), 'mpas-sw-tl-ad_b200', 'csrc')


@pytest.fixture(scope='module')
def exe(tmp_path_factory):
    gxx = shutil.which('g++')
    if not gxx:
        pytest.skip('no g++')
    out = str(tmp_path_factory.mktemp('turns') / 'turns')
    subprocess.run([gxx, '-O2', '-std=c++17', '-pthread', '-I' + CSRC, os.path.join(HERE, 'turns_check.cpp'), '-o', out],
                   check=True)
    return out


@pytest.mark.parametrize('pieces', [0, 1, 2, 3, 16, 64])
@pytest.mark.parametrize('fails_at', [-1, 0, 2])
def test_every_piece_runs_once(exe, pieces, fails_at):
    for bad in [-1] + ([pieces - 1] if pieces and fails_at < 0 else []):
        assert subprocess.run([exe, str(pieces), str(fails_at), str(bad)]).returncode == 0
