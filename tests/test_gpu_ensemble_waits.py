"""A bounded wait that runs out in one member's grouped banded solves: the ensemble's
sync reports MLEGS_ERR_TIMEOUT once and names the member, and the ensemble, started
again at the default limit, agrees with runs of the members alone."""

import pytest

from conftest import rel, small_cfg

pytestmark = pytest.mark.gpu

MLEGS_ERR_TIMEOUT = 105


def test_timeout_is_reported_and_the_ensemble_recovers(lib_built):
    import mlegs_b200 as M
    cfgs = [small_cfg(32, 16, 16), small_cfg(64, 32, 32), small_cfg(48, 16, 32)]
    ens = M.Ensemble(cfgs)

    def start():
        states = []
        for ctx, cfg in zip(ens.contexts, cfgs):
            fs = M.initial_state(ctx, cfg)
            ctx.initialize(*fs)
            states.append(fs)
        return states

    try:
        start()
        ens.step(1, graph=False)
        ens.sync()
        member = ens.contexts[1]
        assert member.lib.mlegs_set_wait_limit(member.c, 1) == 0
        ens.step(1, graph=False)
        with pytest.raises(M.MlegsError) as ei:
            ens.sync()
        assert ei.value.code == MLEGS_ERR_TIMEOUT
        assert str(ei.value).endswith("member 1")
        ens.sync()  # reported once
        for ctx in ens.contexts:
            ctx.sync()
        assert member.lib.mlegs_set_wait_limit(member.c, 0) == 0
        states = start()
        ens.step(2, graph=False)
        ens.sync()
        got = [[f.download() for f in fs] for fs in states]
    finally:
        ens.close()
    for cfg, out in zip(cfgs, got):
        ctx = M.Context(cfg)
        fs = M.initial_state(ctx, cfg)
        ctx.initialize(*fs)
        ctx.step(2)
        for (E, ln), f in zip(out, fs):
            R, rln = f.download()
            # the GEMMs of the two forms sum in different orders: the ensemble test's bound
            assert rel(E, R) < 1e-13 and abs(ln - rln) <= 1e-13 * max(1.0, abs(rln))
        ctx.close()
