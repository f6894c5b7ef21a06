"""Member counts that the sweeps pad to a vector width: every member of an odd-sized batch equals
the same member of a batch that needs no padding, and the caller's rows keep their own length."""
import numpy as np
import pytest

from helpers import rel, setup
from module_sw_mpas import MpasSwModule

pytestmark = pytest.mark.gpu
torch = pytest.importorskip('torch')


@pytest.mark.parametrize('cfg', [dict(), dict(visc2=1e5, drag=True)])
@pytest.mark.parametrize('precision,counts', [(0, [1, 3, 5, 7, 9]), (1, [1, 3, 5, 9, 13, 33])])
def test_odd_member_counts(precision, counts, cfg):
    from mpsw.torch_api import Engine
    m = setup(MpasSwModule(), 3, 'seeded', dt=600.0, **cfg)
    e = Engine(m)
    rng = np.random.default_rng(2)
    B = 40
    du = torch.tensor(rng.standard_normal((int(m.nedges), B)) * 0.1, device='cuda')
    dh = torch.tensor(rng.standard_normal((int(m.ncells), B)), device='cuda')
    w = e.window(3, ckpt_every=2)
    full = w.tl(du, dh, precision) + w.ad(du, dh, precision)
    for n in counts:
        a, b = du[:, :n].contiguous(), dh[:, :n].contiguous()
        part = w.tl(a, b, precision) + w.ad(a, b, precision)
        for x, y in zip(part, full):
            assert x.shape[1] == n
            if precision == 0:
                assert torch.equal(x, y[:, :n])
            else:  # FP32 stencils are compiled with contraction: one rounding between member widths
                assert rel(x.cpu().numpy(), y[:, :n].cpu().numpy()) < 1e-6
