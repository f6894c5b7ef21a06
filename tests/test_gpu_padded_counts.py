"""The member counts that sweeps run with: a sweep tunes its kernels for the padded count, so the tables show
which one it was."""
import ctypes

import numpy as np
import pytest

from helpers import setup
from module_sw_mpas import MpasSwModule

pytestmark = pytest.mark.gpu
torch = pytest.importorskip('torch')


# FP64: even; FP32: to four, from 24 on to eight; six and whole vectors stay
@pytest.mark.parametrize('precision,B,padded,other', [(0, 3, 4, 6), (0, 9, 10, 12), (0, 10, 10, 12), (0, 13, 14, 16), (1, 3, 4, 8),
                                                      (1, 6, 6, 8), (1, 9, 12, 16), (1, 12, 12, 16), (1, 18, 20, 24),
                                                      (1, 21, 24, 20), (1, 25, 32, 24)])
def test_padded_count(precision, B, padded, other):
    from mpsw.torch_api import Engine
    e = Engine(setup(MpasSwModule(), 2, 'seeded', dt=1200.0))
    rng = np.random.default_rng(0)
    e.window(1).tl(torch.tensor(rng.standard_normal((e.nE, B)), device='cuda'),
                   torch.tensor(rng.standard_normal((e.nC, B)), device='cuda'), precision)

    def tuned(n):
        v = (ctypes.c_int * 16)()
        e.h.call('mpsw_window_tuning', precision, n, v)
        return any(v)
    assert tuned(B) and tuned(padded) and not tuned(other)
