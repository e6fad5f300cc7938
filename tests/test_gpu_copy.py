"""COPY (COPY0) of FFF fields whose rows are shorter, as long as and longer than the
8, 16 and 32 lanes, and the 128 entries, that one team copies: kept rows bit for bit,
cleared rows zero, the log term along."""

import numpy as np
import pytest

from conftest import oracle_grid, random_fff, small_cfg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nxchop", [1, 4, 5, 8, 9, 16, 17, 64, 65, 150])
@pytest.mark.parametrize("ntchop", [1, 9])
def test_copy(lib_built, nxchop, ntchop):
    import mlegs_b200 as M
    nx = 16
    while nx < 2 * nxchop:
        nx *= 2
    cfg = small_cfg(34, 16, nx, nrchop=21, ntchop=ntchop, nxchop=nxchop)
    g = oracle_grid(cfg)
    ctx = M.Context(cfg)
    A = random_fff(g, 86, pad=6)  # rows beyond the chop hold something
    A.E = A.E + 1.0
    a = ctx.field(M.FFF).upload(A.E, 0.3, M.FFF)
    b = ctx.field(M.FFF).upload(np.full_like(A.E, 7.0), 9.0, M.FFF)
    for pad in (0, 3):
        ctx.COPY(b, a, pad)
        E, ln = b.download()
        g.chopset(pad)
        R = g.alloc(A.space)
        R.E[...] = A.E
        g.chopdo(R)
        g.chopset(-pad)
        assert np.array_equal(E, R.E) and ln == 0.3
    ctx.close()
