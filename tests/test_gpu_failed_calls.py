"""Transforms and PROJECT on a stream whose capture has been invalidated on the host
(nothing runs on the device): the call returns an error, and the fields keep their
data and their space."""

import ctypes

import numpy as np
import pytest

from conftest import oracle_grid, random_fff, rel, small_cfg

pytestmark = pytest.mark.gpu


class InvalidCapture:
    """The context's stream in a capture that a forbidden call has invalidated."""

    def __init__(self, ctx):
        self.rt = ctypes.CDLL("libcudart.so.12")  # the library's own runtime
        self.s = ctypes.c_void_p(ctx.lib.mlegs_stream(ctx.c))

    def __enter__(self):
        assert self.rt.cudaStreamBeginCapture(self.s, 1) == 0  # thread-local mode
        assert self.rt.cudaStreamSynchronize(self.s) != 0

    def __exit__(self, *exc):
        graph = ctypes.c_void_p()
        assert self.rt.cudaStreamEndCapture(self.s, ctypes.byref(graph)) != 0
        self.rt.cudaGetLastError()


@pytest.fixture(scope="module")
def env(lib_built):
    import mlegs_b200 as M
    cfg = small_cfg(32, 16, 16)
    ctx = M.Context(cfg)
    yield M, ctx, oracle_grid(cfg)
    ctx.close()


def ppp(M, ctx, g, seed):
    from oracle import transforms as T
    A = random_fff(g, seed)
    T.tofp(g, A)
    return ctx.field(M.PPP).upload(A.E, A.LN, A.space)


@pytest.mark.parametrize("call", ["TOFP", "RTRAN", "TOFF"])
def test_transform(env, call):
    M, ctx, g = env
    f = ppp(M, ctx, g, 90) if call == "TOFF" else ctx.field(M.FFF).upload(random_fff(g, 90).E, 0.4, M.FFF)
    run = {"TOFP": lambda x: ctx.TOFP(x), "RTRAN": lambda x: ctx.RTRAN(x, 1), "TOFF": lambda x: ctx.TOFF(x)}[call]
    space = f.space
    E, ln = f.download()
    with InvalidCapture(ctx):
        with pytest.raises(M.MlegsError):
            run(f)
    assert f.space == space
    E2, ln2 = f.download()
    assert np.array_equal(E, E2) and ln == ln2
    h = ctx.field(space).upload(E, ln, space)
    run(h)
    run(f)
    assert f.space == h.space != space
    assert np.array_equal(f.download()[0], h.download()[0])


def test_project(env):
    from oracle import legops as L
    M, ctx, g = env
    fs = [ppp(M, ctx, g, 91 + q) for q in range(3)]
    before = [f.download()[0] for f in fs]
    psi, chi = ctx.field(M.FFF), ctx.field(M.FFF)
    with InvalidCapture(ctx):
        with pytest.raises(M.MlegsError):
            ctx.PROJECT(*fs, psi, chi, 0.0)
    for f, E in zip(fs, before):
        assert f.space == M.PPP
        assert np.array_equal(f.download()[0], E)
    ctx.PROJECT(*fs, psi, chi, 0.0)
    U = []
    for E in before:
        A = g.alloc(M.PPP)
        A.E[...] = E
        U.append(A)
    P, C = L.project(g, *U, 0.0)
    assert rel(psi.download()[0], P.E) < 1e-11 and rel(chi.download()[0], C.E) < 1e-11


def test_an_error_is_reported_once(env):
    """What a refused call leaves in the runtime is not the next call's error."""
    M, ctx, g = env
    f = ctx.field(M.FFF).upload(random_fff(g, 95).E, 0.4, M.FFF)
    with InvalidCapture(ctx) as _:
        with pytest.raises(M.MlegsError):
            ctx.TOFP(f)
        assert ctypes.CDLL("libcudart.so.12").cudaPeekAtLastError() == 0
    ctx.TOFP(f)
    ctx.sync()
