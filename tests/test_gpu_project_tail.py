"""PROJECT's closing passes (VEL2PLN on PSI's (0, 0) column, the far-field fix, RUP's
line) against the oracle, each LN form, on grids with odd numbers of rows, half
rows and axial modes.  The line has a far field (RUP tends to a constant), so the
log term is of the size of the data.  Tolerance: that of PROJECT's other
comparisons with the oracle."""

import pytest

from conftest import oracle_grid, random_fff, rel, small_cfg

pytestmark = pytest.mark.gpu

GRIDS = {
    "32x16x16": dict(),
    "34x16x32": dict(nrchop=27),                              # odd NRH, NRCHOP
    "66x32x16": dict(nrchop=41, ntchop=13, nxchop=7),         # odd axial modes
    "128x32x64": dict(),
}


@pytest.mark.parametrize("form", ["none", "value", "psi"])
@pytest.mark.parametrize("name", list(GRIDS))
def test_project_tail(lib_built, name, form):
    import mlegs_b200 as M
    from oracle import legops as L
    from oracle import transforms as T
    nr, nth, nx = (int(v) for v in name.split("x"))
    cfg = small_cfg(nr, nth, nx, **GRIDS[name])
    g = oracle_grid(cfg)
    U = [random_fff(g, 20 + q, decay=4.0) for q in range(3)]
    for F in U:
        T.rtran(g, F, 1)
    U[1].E[:g.NR, 0, 0] += 2.0 * (1.0 + g.X[:g.NR])
    ln = {"none": None, "value": 0.25, "psi": "psi"}[form]
    ctx = M.Context(cfg)
    fs = [ctx.field(u.space).upload(u.E, 0.0, u.space) for u in U]
    psi, chi = ctx.field(M.FFF), ctx.field(M.FFF)
    ctx.PROJECT(*fs, psi, chi, ln)
    P, W = L.project(g, *U, ln)
    E, lnp = psi.download()
    assert rel(E, P.E) < 1e-11
    assert abs(lnp - P.LN) < 1e-11 * max(1.0, abs(P.LN))
    E, lnc = chi.download()
    assert rel(E, W.E) < 1e-11 and lnc == 0.0
    for f, u in zip(fs, U):
        assert rel(f.download()[0], u.E) < 1e-11
    ctx.close()
