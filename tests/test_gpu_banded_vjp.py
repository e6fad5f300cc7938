"""The transposed IHELM solves out of place (a step VJP's three in one launch) against
the in-place operator TRANSPOSE("IHELM"), for columns in shared memory and columns
too long for it (more than 727 rows).

The VJP's history cotangents are those of the solved state alone:
n_bar = -dt/2 (-ALP IHELM^T(bar)), ALP = 2 / (NU dt), so they are the in-place
solve times dt ALP / 2 up to a handful of roundings."""

import numpy as np
import pytest

from conftest import oracle_grid, random_fff, rel, small_cfg

pytestmark = pytest.mark.gpu

# nr, nth, nx, nrchop, ntchop, nxchop: 58 rows, 727 (the last in shared memory), 728, 844
GRIDS = [(64, 16, 16, 58, 5, 4), (734, 16, 16, 727, 2, 2), (736, 16, 16, 728, 2, 2), (850, 16, 16, 844, 2, 2)]


@pytest.mark.parametrize("dims", GRIDS)
def test_step_vjp_solves_match_the_single_transpose(lib_built, dims):
    import mlegs_b200 as M
    nr, nth, nx, nrchop, ntchop, nxchop = dims
    cfg = small_cfg(nr, nth, nx, nrchop=nrchop, ntchop=ntchop, nxchop=nxchop, nu=1e-3, kappa=3e-3)
    g = oracle_grid(cfg)
    ctx = M.Context(cfg)

    def up(F):
        return ctx.field(M.FFF).upload(F.E, F.LN, F.space)

    def fff(seed, ln=0.0):
        F = random_fff(g, seed)
        F.LN = ln
        return F

    state = [up(fff(40 + q)) for q in range(3)]
    bars = [fff(50, 0.3), fff(51, -0.2)] + [fff(52 + q) for q in range(4)]
    # what the pool's temporaries hold before the call has no part in its result
    for seed in (70, 71):
        junk = [up(fff(seed + 10 * q, 1.0)) for q in range(3)]
        ctx.AB2_STEP_VJP(junk, [up(fff(seed + q)) for q in range(6)], [ctx.field(M.FFF) for _ in range(6)])
    outs = [ctx.field(M.FFF) for _ in range(6)]
    ctx.AB2_STEP_VJP(state, [up(F) for F in bars], outs)
    for q, nu in enumerate((cfg.nu, cfg.nu, cfg.kappa)):
        alp = 2 / (nu * cfg.dt)
        x = ctx.field(M.FFF)
        ctx.TRANSPOSE("IHELM", [up(bars[q])], [x], 0, alp)
        X, _ = x.download()
        E, _ = outs[3 + q].download()
        assert np.abs(X).max() > 0
        # four roundings of 1.1e-16 (the two scalings, ALP and dt ALP / 2)
        assert rel(E, 0.5 * cfg.dt * alp * X) < 1e-14
    ctx.close()
