"""TOFP of several fields in groups of fewer than all (the form of grids whose PFF images
would take more than 8 GiB) against one launch for all, bit for bit: images used again
by the next group, on one stream (FP64) and on two (split-BF16, three fields in flight)."""

import numpy as np
import pytest

from conftest import small_cfg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("adams", [True, False])
def test_groups_agree(lib_built, split, adams):
    import mlegs_b200 as M
    cfg = small_cfg(64, 32, 64, adams=adams)
    ctx = M.Context(cfg, precision=M.PREC_SPLIT, split_slices=6) if split else M.Context(cfg)
    ref = None
    for n in (10, 6, 5, 4, 3, 2, 1):
        assert ctx.lib.mlegs_tofp_group(ctx.c, n) == n
        fs = M.initial_state(ctx, cfg)
        outs = [ctx.field(M.FFF) for _ in range(3)]
        ctx.CALC_BOUSSI_FORCE(*fs, *outs)
        ctx.initialize(*fs)
        ctx.step(2)
        got = [f.download() for f in outs + list(fs)]
        if ref is None:
            ref = got
        for (E, ln), (R, rln) in zip(got, ref):
            assert np.array_equal(E, R) and ln == rln
    ctx.close()


def test_images_of_a_large_full_spectrum_grid(lib_built):
    """128 x 512 x 1024 without dealiasing, 1.07 GB an image: no more of them than three
    field buffers (the context takes about 41 GB)."""
    import mlegs_b200 as M
    cfg = small_cfg(128, 512, 1024, nrchop=85, ntchop=512, nxchop=512)
    ctx = M.Context(cfg)
    image = 512 * 128 * 1023
    assert ctx.lib.mlegs_tofp_group(ctx.c, 0) * image <= 3 * 128 * 512 * 1024
    assert ctx.lib.mlegs_tofp_group(ctx.c, 10) == 3
    assert ctx.lib.mlegs_tofp_group(ctx.c, -1) == -1
    ctx.close()
