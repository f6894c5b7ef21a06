"""Member counts that are padded run unpadded where device memory is too short for the padding."""
import numpy as np
import pytest

from helpers import setup
from module_sw_mpas import MpasSwModule

pytestmark = pytest.mark.gpu
torch = pytest.importorskip('torch')


@pytest.mark.parametrize('precision,B,tol', [(1, 5, 1e-6), (0, 3, 0.0)])
def test_count_runs_unpadded_when_memory_is_short(precision, B, tol):
    from mpsw.torch_api import Engine
    rng = np.random.default_rng(0)

    def window():
        e = Engine(setup(MpasSwModule(), 6, 'seeded', dt=150.0))
        x = (torch.tensor(rng.standard_normal((e.nE, B)), device='cuda'), torch.tensor(rng.standard_normal((e.nC, B)), device='cuda'))
        return e, x, e.window(1, storage=0)

    def sweep(e, x, w):
        a, b = e.to_internal(x[0], 1), e.to_internal(x[1], 0)
        free = torch.cuda.mem_get_info()[0]
        w.tl_internal(a, b, precision)
        torch.cuda.synchronize()
        return a, b, free - torch.cuda.mem_get_info()[0]
    e, x, w = window()
    u, h, padded = sweep(e, x, w)
    e2, _, w2 = window()
    torch.cuda.empty_cache()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - int(0.9 * padded), dtype=torch.uint8, device='cuda')
    try:
        got = sweep(e2, x, w2)
    finally:
        del hold
        torch.cuda.empty_cache()
    assert got[2] < 0.9 * padded
    for a, b in zip(got, (u, h)):  # (a width of one member: the same sums, FP32 ones contracted differently)
        assert float((a - b).norm()) <= tol * float(b.norm())
