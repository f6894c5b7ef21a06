"""Large host copies over threads (csrc/mpsw_parts.h): memory that runs out while the threads are started
leaves the copy whole and the process alive."""
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
    out = str(tmp_path_factory.mktemp('parts') / 'parts')
    subprocess.run([gxx, '-O2', '-std=c++17', '-pthread', '-I' + CSRC, os.path.join(HERE, 'parts_check.cpp'), '-o', out],
                   check=True)
    return out


@pytest.mark.parametrize('fails_at', [-1, 0, 1, 2, 3, 4, 5])
def test_copy_survives_a_failed_allocation(exe, fails_at):
    assert subprocess.run([exe, str(fails_at)]).returncode == 0
