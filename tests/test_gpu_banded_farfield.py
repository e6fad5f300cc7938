"""The far-field fix (CALCAT1) that IDEL2LN and IDEL2 end with, in both forms of the
solves (up to 727 rows in shared memory, beyond in global memory): the m = 0 columns
vanish at infinity."""

import numpy as np
import pytest

from conftest import oracle_grid, random_fff, small_cfg

pytestmark = pytest.mark.gpu

# nr, nrchop: row counts on either side of the forms' limit and of the sum's 32-row runs
ROWS = [(64, 58), (734, 727), (736, 728), (744, 736), (850, 844)]


@pytest.mark.parametrize("nr,nrchop", ROWS)
def test_columns_vanish_at_infinity(lib_built, nr, nrchop):
    import mlegs_b200 as M
    cfg = small_cfg(nr, 16, 16, nrchop=nrchop, ntchop=2, nxchop=3)
    g = oracle_grid(cfg)
    ctx = M.Context(cfg)
    B = random_fff(g, 85)
    b = ctx.field(M.FFF).upload(B.E, 0.3, B.space)
    for call in (lambda a: ctx.IDEL2LN(b, a), lambda a: ctx.IDEL2(b, a), lambda a: ctx.IDEL2(b, a, LN=0.7)):
        a = ctx.field(M.FFF)
        call(a)
        E, _ = a.download()
        terms = g.AT1[:nrchop, None] * E[:nrchop, 0, :]
        assert np.abs(terms).sum() > 0
        # a sum of nrchop rounded terms: nrchop roundings of 1.1e-16
        assert (np.abs(terms.sum(0)) <= nrchop * 1.2e-16 * np.abs(terms).sum(0)).all()
    ctx.close()
