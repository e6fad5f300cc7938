"""Transforms and the right-hand side at the sizes where their launches change form,
against the oracle: VERFFT's warps per block (2, 4 and 8 by the number of azimuthal
modes, at every NX of the four-step kernels), the theta stage's lines per warp (two up
to NTH = 32) and its last, partly filled round of lines, and radial sizes beyond the
bulk GEMMs (NRH > 128)."""

import pytest

from conftest import oracle_grid, oracle_physics, random_fff, rel, small_cfg

pytestmark = pytest.mark.gpu


def mode_counts(nx):
    lines = 32 // {16: 4, 32: 4, 64: 8, 128: 8, 256: 16, 512: 16}[nx]  # of a warp
    return [2 * lines, 2 * lines + 1, 4 * lines, 4 * lines + 1]


@pytest.mark.parametrize("nx,ntchop", [(nx, nt) for nx in (16, 32, 64, 128, 256, 512) for nt in mode_counts(nx)])
def test_transforms(lib_built, nx, ntchop):
    import mlegs_b200 as M
    from oracle import transforms as T
    cfg = small_cfg(18, 64, nx, ntchop=ntchop)
    g = oracle_grid(cfg)
    A = random_fff(g, 120)
    ctx = M.Context(cfg)
    f = ctx.field(M.FFF).upload(A.E, 0.2, M.FFF)
    A.LN = 0.2
    ctx.TOFP(f)
    T.tofp(g, A)
    assert rel(f.download()[0], A.E) < 1e-12
    ctx.TOFF(f)
    T.toff(g, A)
    assert rel(f.download()[0], A.E) < 1e-12
    ctx.close()


@pytest.mark.parametrize("dims", [(34, 16, 16), (34, 32, 16), (34, 64, 16), (34, 128, 16), (34, 256, 16),
                                  (18, 512, 16), (264, 16, 16)])
def test_force(lib_built, dims):
    import mlegs_b200 as M
    from mlegs_b200.inputs import perturbation_coefficients
    from oracle import boussinesq as BQ
    from oracle import layout
    cfg = small_cfg(*dims, nrchop=min(2 * dims[0] // 3, 60), ntchop=min(2 * dims[1] // 3, 21))
    g = oracle_grid(cfg)
    S = layout.initial_state(g, *[perturbation_coefficients(cfg, i) for i in range(3)])
    ctx = M.Context(cfg)
    fs = [ctx.field(M.FFF).upload(F.E, F.LN, F.space) for F in S]
    outs = [ctx.field(M.FFF) for _ in range(3)]
    ctx.CALC_BOUSSI_FORCE(*fs, *outs)
    for o, R in zip(outs, BQ.calc_boussi_force(g, oracle_physics(cfg), *[F.copy() for F in S])):
        E, ln = o.download()
        # the bounds of the right-hand side's other comparisons with the oracle
        assert rel(E, R.E) < 1e-10
        assert abs(ln - R.LN) < 1e-10 * max(1.0, abs(R.LN))
    ctx.close()
