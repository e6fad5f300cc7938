"""PC2VEL, PC2VOR and GRAD on the smallest grids, whose FFF fields have 4 to 10 entries
(a launch clears nine log-term slots): against the oracle, into fields whose log
terms held something before."""

import pytest

from conftest import oracle_grid, random_fff, rel, small_cfg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,nrchop", [(4, 3), (6, 3), (8, 4), (10, 4)])
def test_derivative_operators(lib_built, nr, nrchop):
    import mlegs_b200 as M
    from oracle import legops as L
    cfg = small_cfg(nr, 16, 16, nrchop=nrchop, ntchop=1, nxchop=1)
    g = oracle_grid(cfg)
    ctx = M.Context(cfg)
    P, C = random_fff(g, 60), random_fff(g, 61)
    P.LN, C.LN = 0.4, -0.7
    psi, chi = (ctx.field(M.FFF).upload(F.E, F.LN, F.space) for F in (P, C))
    junk = random_fff(g, 62)
    for dev, ref in ((ctx.PC2VEL, L.pc2vel), (ctx.PC2VOR, L.pc2vor), (ctx.GRAD, lambda g_, a, _: L.grad(g_, a))):
        outs = [ctx.field(M.FFF).upload(junk.E, 3.5, junk.space) for _ in range(3)]
        if dev == ctx.GRAD:
            ctx.GRAD(psi, *outs)
        else:
            dev(psi, chi, *outs)
        for o, R in zip(outs, ref(g, P, C)):
            E, ln = o.download()
            assert ln == R.LN == 0.0
            assert rel(E, R.E) < 1e-12
    ctx.close()
