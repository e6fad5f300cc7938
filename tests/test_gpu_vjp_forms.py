"""The forms of the right-hand side and of its reverse that a grid or the physics select:
the step VJP with and without its joint solves (KAPPA = 0), CALC_BOUSSI_FORCE's VJP in
joint launches and operator by operator (NX below the batched FFTs, NRH above the bulk
GEMMs), against the oracle; and CALC_BOUSSI_FORCE into its own inputs, in the forms with
and without PROJECT's closing passes in the solve, against separate outputs."""

import numpy as np
import pytest

from conftest import oracle_grid, oracle_physics, random_fff, rel, small_cfg

pytestmark = pytest.mark.gpu

VJP = {
    "joint, odd half and chops": ((66, 32, 16), dict(nrchop=41, ntchop=13, nxchop=7)),
    "kappa 0": ((48, 32, 32), dict(kappa=0.0)),
    "kappa 0, NX 8": ((48, 16, 8), dict(kappa=0.0)),
    "NX 8": ((48, 16, 8), dict()),
    "NRH 132": ((264, 16, 16), dict(nrchop=40, ntchop=5, nxchop=5)),
}


@pytest.mark.parametrize("name", list(VJP))
def test_step_vjp(lib_built, name):
    import mlegs_b200 as M
    from mlegs_b200.inputs import perturbation_coefficients
    from oracle import adjoint as AD
    from oracle import boussinesq as BQ
    from oracle import layout
    dims, kw = VJP[name]
    cfg = small_cfg(*dims, **kw)
    g = oracle_grid(cfg)
    s = BQ.Solver(g, oracle_physics(cfg),
                  *layout.initial_state(g, *[perturbation_coefficients(cfg, i) for i in range(3)]))
    s.initialize()
    ctx = M.Context(cfg)

    def up(F):
        return ctx.field(F.space).upload(F.E, F.LN, F.space)

    bars = {}
    for i, k in enumerate(AD.AB2_STATE):
        bars[k] = random_fff(g, 110 + i)
        bars[k].LN = 0.1 * (i + 1) if k in ("psi", "chi", "n_psi", "n_chi") else 0.0
    ref = AD.ab_cn_step_vjp(s, bars)
    state = [up(getattr(s, k)) for k in ("psi", "chi", "b")]
    outs = [ctx.field() for _ in AD.AB2_STATE]
    ctx.AB2_STEP_VJP(state, [up(bars[k]) for k in AD.AB2_STATE], outs)
    for o, k in zip(outs, AD.AB2_STATE):
        E, ln = o.download()
        # the bounds of the step VJP's other comparison with the oracle
        assert rel(E, ref[k].E) < 1e-10, k
        assert abs(ln - ref[k].LN) <= 1e-10 * max(np.abs(ref[k].E).max(), abs(ref[k].LN)), k
    ctx.close()


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("dims", [(64, 32, 32), (16, 16, 16)])
@pytest.mark.parametrize("order", [(0, 1, 2), (2, 0, 1)])
def test_force_into_its_inputs(lib_built, dims, split, order):
    import mlegs_b200 as M
    cfg = small_cfg(*dims)
    ctx = M.Context(cfg, precision=M.PREC_SPLIT, split_slices=6) if split else M.Context(cfg)
    a, b = M.initial_state(ctx, cfg), M.initial_state(ctx, cfg)
    for q, f in enumerate(a):  # log terms of their own
        E, _ = f.download()
        for h in (f, b[q]):
            h.upload(E, 0.2 * (q + 1), M.FFF)
    outs = [ctx.field(M.FFF) for _ in range(3)]
    ctx.CALC_BOUSSI_FORCE(*a, *outs)
    ctx.CALC_BOUSSI_FORCE(*b, *[b[q] for q in order])
    for o, q in zip(outs, order):
        (E, ln), (R, rln) = b[q].download(), o.download()
        assert np.array_equal(E, R) and ln == rln
    ctx.close()
