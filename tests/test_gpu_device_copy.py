"""DEVICE_COPY between fields and the caller's buffers in every form it takes: this
device's memory (one launch; up to the last byte of its allocation), buffers that are
only 8-byte aligned and managed memory (the runtime's copies); with and without a log
term; every space."""

import ctypes

import numpy as np
import pytest

from conftest import oracle_grid, small_cfg

pytestmark = pytest.mark.gpu


class Buffer:
    """nbytes of device memory from the runtime, at `offset` bytes into an allocation
    that ends with it."""

    def __init__(self, nbytes, offset=0, managed=False):
        self.rt = ctypes.CDLL("libcudart.so.12")
        self.base = ctypes.c_void_p()
        self.nbytes = nbytes
        size = ctypes.c_size_t(nbytes + offset)
        if managed:
            assert self.rt.cudaMallocManaged(ctypes.byref(self.base), size, 1) == 0
        else:
            assert self.rt.cudaMalloc(ctypes.byref(self.base), size) == 0
        self.ptr = self.base.value + offset

    def _copy(self, dst, src):
        assert self.rt.cudaMemcpy(ctypes.c_void_p(dst), ctypes.c_void_p(src), ctypes.c_size_t(self.nbytes), 4) == 0

    def put(self, a):
        self._copy(self.ptr, a.ctypes.data)
        return self

    def get(self):
        a = np.empty(self.nbytes // 8)
        self._copy(a.ctypes.data, self.ptr)
        return a

    def free(self):
        self.rt.cudaFree(self.base)


@pytest.mark.parametrize("form", [(0, False), (512, False), (8, False), (0, True)],
                         ids=["aligned", "offset", "unaligned", "managed"])
@pytest.mark.parametrize("with_ln", [True, False])
def test_round_trip(lib_built, form, with_ln):
    import mlegs_b200 as M
    cfg = small_cfg(34, 16, 16)
    g = oracle_grid(cfg)
    ctx = M.Context(cfg)
    rng = np.random.default_rng(5)
    nt, nk = min(cfg.ntchop, cfg.nth), 2 * cfg.nxchop - 1
    elems = {M.FFF: nt * g.NRCHOPDIM * nk, M.PFF: nt * cfg.nr * nk, M.PFP: nt * cfg.nr * cfg.nx,
             M.PPP: cfg.nth * cfg.nr * cfg.nx}
    for space, n in elems.items():
        a = rng.standard_normal(2 * n)
        src, dst = (Buffer(16 * n, *form) for _ in range(2))
        lns, lnd = Buffer(8).put(np.array([0.75])), Buffer(8).put(np.array([-1.0]))
        f = ctx.field(M.FFF).upload(np.zeros(ctx.shape(M.FFF), complex), 2.5, M.FFF)
        src.put(a)
        ctx.DEVICE_COPY(f, True, space, src.ptr, lns.ptr if with_ln else None)
        assert f.space == space
        ctx.DEVICE_COPY(f, False, space, dst.ptr, lnd.ptr if with_ln else None)
        ctx.sync()
        assert np.array_equal(dst.get(), a)
        assert lnd.get()[0] == (0.75 if with_ln else -1.0)
        assert f.download()[1] == (0.75 if with_ln else 0.0)
        for b in (src, dst, lns, lnd):
            b.free()
    ctx.close()
