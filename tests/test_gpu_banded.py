"""The banded solves at the edges of their blocks (16 systems, 8 rows a chunk):
system sizes and axial mode counts on either side of a multiple, a single
axial mode, results in place, and columns too long for shared memory."""

import numpy as np
import pytest

from conftest import oracle_grid, random_fff, rel, small_cfg

pytestmark = pytest.mark.gpu

# nr, nth, nx, nrchop, ntchop, nxchop
GRIDS = [(32, 16, 32, 24, 5, 8), (32, 16, 32, 25, 30, 9), (40, 16, 16, 31, 7, 1), (96, 16, 64, 88, 4, 17)]


def grid(nr, nth, nx, nrchop, ntchop, nxchop):
    cfg = small_cfg(nr, nth, nx, nrchop=nrchop, ntchop=ntchop, nxchop=nxchop)
    return cfg, oracle_grid(cfg)


@pytest.mark.parametrize("dims", GRIDS)
@pytest.mark.parametrize("inplace", [False, True])
def test_solves(lib_built, dims, inplace):
    import mlegs_b200 as M
    from oracle import legops as L
    cfg, g = grid(*dims)
    ctx = M.Context(cfg)
    for q, (dev, ref) in enumerate([
            (lambda b, a: ctx.IDEL2LN(b, a), lambda B: L.idel2ln(g, B)),
            (lambda b, a: ctx.IDEL2(b, a), lambda B: L.idel2(g, B)),
            (lambda b, a: ctx.IDEL2(b, a, LN=0.7), lambda B: L.idel2(g, B, 0.7)),
            (lambda b, a: ctx.IHELM(b, a, 350.0), lambda B: L.ihelm(g, B, 350.0))]):
        B = random_fff(g, 20 + q)
        B.LN = 0.3
        b = ctx.field(M.FFF).upload(B.E, B.LN, B.space)
        a = b if inplace else ctx.field(M.FFF)
        dev(b, a)
        E, ln = a.download()
        R = ref(B)
        assert rel(E, R.E) < 1e-10
        assert abs(ln - R.LN) < 1e-10 * max(1.0, abs(R.LN))
    ctx.close()


def test_long_columns(lib_built):
    """844 rows: the column no longer fits in shared memory."""
    import mlegs_b200 as M
    from oracle import legops as L
    cfg, g = grid(850, 16, 16, 844, 2, 2)
    ctx = M.Context(cfg)
    B = random_fff(g, 31)
    B.LN = 0.3
    b = ctx.field(M.FFF).upload(B.E, B.LN, B.space)
    a = ctx.field(M.FFF)
    ctx.IHELM(b, a, 2.0e6)
    R = L.ihelm(g, B, 2.0e6)
    E, ln = a.download()
    # DEL2's entries grow as n^2 (n^4 in the condition number): 1e-16 (844^4 / 2e6)
    assert rel(E, R.E) < 1e-9 and abs(ln - R.LN) < 1e-12
    # IHELM^T against IHELM by the dot-product identity
    Y = random_fff(g, 32)
    y = ctx.field(M.FFF).upload(Y.E, 0.0, Y.space)
    x = ctx.field(M.FFF)
    ctx.TRANSPOSE("IHELM", [y], [x], 0, 2.0e6)
    X, xln = x.download()
    lhs = np.vdot(Y.E, E).real
    rhs = np.vdot(X, B.E).real + xln * B.LN
    assert abs(lhs - rhs) < 1e-9 * np.linalg.norm(Y.E) * np.linalg.norm(E)
    ctx.close()
