"""A NaN in the state reaches the entities whose stencils hold it, as in the oracle, and no others: the
padded slots of a tile's records (pentagons have five edges, their edges nine neighbours) read a neighbour
that the entity has anyway."""
import numpy as np
import pytest

import oracle as O
from helpers import setup
from test_stage_tiles import lib, run  # noqa: F401

NAMES = ['tend_u', 'tend_h', 'u', 'h_edge', 'v', 'gradpvt', 'gradpvn', 'pv_edge', 'vorticity', 'h_vertex', 'ke']


@pytest.mark.parametrize('phys', [dict(), dict(visc2=2e5, visc4=1e15, drag=True, wind=True)])
@pytest.mark.parametrize('var', ['u', 'h'])
def test_nan_stays_in_its_stencils(lib, var, phys):  # noqa: F811
    o = setup(O.OracleModule(), 1, 'seeded', **phys)
    clean = getattr(o, var)[0, 0].copy()
    for i in range(clean.size):
        x = clean.copy()
        x[i] = np.nan
        getattr(o, var)[0, 0] = x
        outs, _ = run(lib, o, 5)
        o.solve_diagnostics()
        o.compute_tend()
        for n, a in zip(NAMES, outs):
            assert np.array_equal(np.isnan(a), np.isnan(np.asarray(getattr(o, n))[0].ravel())), (i, n)
