"""The banded solves' bounded waits: a context with a wait limit of one SM cycle
reports MLEGS_ERR_TIMEOUT once at its next sync, and computes the oracle's solution
again at the default limit.  Sizes: fewer chunks than the ring holds (the copying warp
has issued everything when the solving one stops), more, the 7-band system, and
columns in global memory."""

import pytest

from conftest import oracle_grid, random_fff, rel, small_cfg

pytestmark = pytest.mark.gpu

MLEGS_ERR_TIMEOUT = 105
GRIDS = [(32, 16, 16, 12, 4, 4), (64, 16, 32, 58, 5, 9), (736, 16, 16, 728, 2, 2)]


@pytest.mark.parametrize("op", ["IDEL2LN", "IHELM", "IHELM_T"])
@pytest.mark.parametrize("dims", GRIDS)
def test_wait_runs_out_and_context_recovers(lib_built, dims, op):
    import mlegs_b200 as M
    from oracle import legops as L
    nr, nth, nx, nrchop, ntchop, nxchop = dims
    cfg = small_cfg(nr, nth, nx, nrchop=nrchop, ntchop=ntchop, nxchop=nxchop)
    g = oracle_grid(cfg)
    alp = 2.0e6
    ctx = M.Context(cfg)
    B = random_fff(g, 80)
    b, a = ctx.field(M.FFF).upload(B.E, 0.2, B.space), ctx.field(M.FFF)
    B.LN = 0.2

    def call():
        if op == "IDEL2LN":
            ctx.IDEL2LN(b, a)
        elif op == "IHELM":
            ctx.IHELM(b, a, alp)
        else:
            ctx.TRANSPOSE("IHELM", [b], [a], 0, alp)
        ctx.sync()

    call()  # the factors exist
    before, ln = a.download()
    assert ctx.lib.mlegs_set_wait_limit(ctx.c, 1) == 0
    with pytest.raises(M.MlegsError) as ei:
        call()
    assert ei.value.code == MLEGS_ERR_TIMEOUT
    ctx.sync()  # reported once
    assert ctx.lib.mlegs_set_wait_limit(ctx.c, 0) == 0
    call()
    E, ln2 = a.download()
    assert (E == before).all() and ln2 == ln
    if op == "IHELM":
        R = L.ihelm(g, B, alp)
        assert rel(E, R.E) < 1e-9  # as for the long columns of the banded solves' test
    ctx.close()
