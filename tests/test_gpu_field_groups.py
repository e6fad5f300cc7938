"""CALC_BOUSSI_FORCE and the AB2-CN step on the grids where their launches
change form, against the oracle: all fields in one launch per transform stage
(small PFF images) or groups of three on two streams (images over 8 MiB), NR
whose half is odd (no bulk-copy RTRAN: one launch per field), the banded
solves below and above 72 rows, and KAPPA = 0 (the step without the joint
viscous solves)."""

import pytest

from conftest import oracle_grid, oracle_physics, rel, small_cfg

pytestmark = pytest.mark.gpu

GRIDS = {
    "32x16x16": dict(),
    "34x16x32_odd_half": dict(),
    "66x32x16_odd_half_chops": dict(nrchop=41, ntchop=13, nxchop=7),
    "100x64x32_chops": dict(nrchop=61, ntchop=37, nxchop=11),
    "128x32x64": dict(),                     # more than 72 rows
    "192x64x128": dict(),                    # PFF image 10.7 MB
}


def config(name, **kw):
    nr, nth, nx = (int(v) for v in name.split("_")[0].split("x"))
    return small_cfg(nr, nth, nx, **dict(GRIDS[name], **kw))


@pytest.mark.parametrize("name", list(GRIDS))
def test_force_and_ab2_step(lib_built, name):
    import mlegs_b200 as M
    from mlegs_b200.inputs import perturbation_coefficients
    from oracle import boussinesq as BQ
    from oracle import layout
    cfg = config(name)
    g = oracle_grid(cfg)
    P, C, B = layout.initial_state(g, *[perturbation_coefficients(cfg, i) for i in range(3)])
    ctx = M.Context(cfg)
    fs = []
    for F in (P, C, B):
        fs.append(ctx.field(M.FFF).upload(F.E, F.LN, F.space))
    outs = [ctx.field(M.FFF) for _ in range(3)]
    ctx.CALC_BOUSSI_FORCE(*fs, *outs)
    ref = BQ.calc_boussi_force(g, oracle_physics(cfg), P.copy(), C.copy(), B.copy())
    for o, R in zip(outs, ref):
        E, ln = o.download()
        assert rel(E, R.E) < 1e-10
        assert abs(ln - R.LN) < 1e-10 * max(1.0, abs(R.LN))
    s = BQ.Solver(g, oracle_physics(cfg), P, C, B)
    s.initialize()
    s.step()
    ctx.initialize(*fs)
    ctx.step(1)
    for f, R in zip(fs, (s.psi, s.chi, s.b)):
        E, ln = f.download()
        assert rel(E, R.E) < 1e-10
        assert abs(ln - R.LN) < 1e-10 * max(1.0, abs(R.LN))
    ctx.close()


@pytest.mark.parametrize("kappa", [0.0, 3e-3])
def test_ab2_steps_with_own_diffusivity(lib_built, kappa):
    import mlegs_b200 as M
    from mlegs_b200.inputs import perturbation_coefficients
    from oracle import boussinesq as BQ
    from oracle import layout
    cfg = config("66x32x16_odd_half_chops", kappa=kappa)
    g = oracle_grid(cfg)
    s = BQ.Solver(g, oracle_physics(cfg),
                  *layout.initial_state(g, *[perturbation_coefficients(cfg, i) for i in range(3)]))
    s.initialize()
    ctx = M.Context(cfg)
    fs = M.initial_state(ctx)
    ctx.initialize(*fs)
    for _ in range(3):
        s.step()
    ctx.step(3, graph=True)
    for f, R in zip(fs, (s.psi, s.chi, s.b)):
        E, ln = f.download()
        assert rel(E, R.E) < 1e-10
        assert abs(ln - R.LN) < 1e-10 * max(1.0, abs(R.LN))
    ctx.close()
