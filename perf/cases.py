"""Timed cases of the library: what its users have it do, through the Python
binding's public entry points, over the range of grids they run.

Kinds (each is one call sequence of a host program; sizes are the case's):

  roundtrip  COPY, TOFP, TOFF of one field: FFF -> PPP -> FFF, the transform
             pair around any work in physical space (FP64, or the split-BF16
             form of the Legendre GEMMs).
  rhs        CALC_BOUSSI_FORCE: the right-hand side of the AB2-CN step.
  project    PROJECT of a velocity-form vector given as physical samples: the
             physical-to-spectral direction with the solenoidal projection.
  operators  PC2VEL, PC2VOR and GRAD: the velocity, vorticity and gradient of a
             state, as diagnostics and the right-hand sides need them.
  solves     IDEL2LN, IDEL2 and IHELM: the banded systems of a step.
  ab2        steady AB2-CN steps of a run, replayed as a CUDA graph.
  etd        steady ETD2AB-CN steps (hyperviscosity), replayed as a graph.
  vjp        the reverse mode of one AB2-CN step on torch tensors.
  ensemble   several independent AB2-CN runs of different grids in lock-step.

Fields are handed over and come back in the device layout ([m][n][k] for FFF,
[r][z][j] for PPP) through DEVICE_COPY, as the gradient path does.
"""

import math

import numpy as np
import torch

import mlegs_b200 as M
from mlegs_b200.adjoint import DeviceAB2
from mlegs_b200.inputs import CONFIGS, Config, chops, ensemble_configs


def _case(kind, nr, nth, nx, nrchop=None, ntchop=None, nxchop=None, **kw):
    c = chops(nr, nth, nx)
    return dict(kind=kind, nr=nr, nth=nth, nx=nx, nrchop=nrchop or c[0], ntchop=ntchop or c[1],
                nxchop=nxchop or c[2], **kw)


def listed():
    def named(name, c):
        return dict(c, name=name)

    return [
        # the smallest grid of the batched runs: a call is a handful of launches
        named("roundtrip_48x32x32", _case("roundtrip", 48, 32, 32)),
        # the transform workload at its full size
        named("roundtrip_256x256x256", _case("roundtrip", 256, 256, 256)),
        # the same pair with the split-BF16 Legendre GEMMs at the flagship grid
        named("roundtrip_split_192x128x256", _case("roundtrip", 192, 128, 256, split=6)),
        # the right-hand side at the AB2-CN IVP grid (chops as that configuration gives them)
        named("rhs_64x32x32", _case("rhs", 64, 32, 32, 58, 16, 16)),
        # the right-hand side at a mid-size grid with odd chops
        named("rhs_100x64x128", _case("rhs", 100, 64, 128, 61, 37, 41)),
        # projection of physical samples at a batched-run grid
        named("project_128x64x128", _case("project", 128, 64, 128)),
        # velocity, vorticity and gradient with ragged chops
        named("operators_130x128x128", _case("operators", 130, 128, 128, 83, 71, 39)),
        # the banded systems of the flagship grid
        named("solves_192x128x256", _case("solves", 192, 128, 256)),
        # a short AB2-CN run of the IVP: ten replayed steps, latency-bound
        named("ab2_64x32x32", _case("ab2", 64, 32, 32, 58, 16, 16, steps=10)),
        # one step of the flagship run
        named("etd_192x128x256", _case("etd", 192, 128, 256, steps=1)),
        # one reverse step of the gradient configuration
        named("vjp_96x64x64", _case("vjp", 96, 64, 64)),
        # sixteen runs of uneven grids, one lock-step step
        named("ensemble_16", dict(kind="ensemble", runs=16, grids=2024, steps=1)),
    ]


def draw(rng):
    kind = rng.choice(["roundtrip", "roundtrip", "rhs", "rhs", "project", "operators", "solves", "ab2", "ab2", "etd", "etd",
                       "vjp", "ensemble"])
    if kind == "ensemble":
        return dict(kind="ensemble", runs=rng.randint(4, 16), grids=rng.randrange(1 << 20), steps=rng.choice([1, 2]))
    top = 96 * 64 * 64 if kind == "vjp" else 192 * 128 * 256
    while True:
        nr = 2 * int(round(math.exp(rng.uniform(math.log(16), math.log(128)))))
        nth = 2 ** rng.randint(4, 8)
        nx = 2 ** rng.randint(4, 8)
        if nr * nth * nx <= top:
            break
    # the 2/3 rule, or fewer modes than that allows (odd counts among them)
    c = [v if rng.random() < 0.3 else max(8 if i == 0 else 3, int(round(v * rng.uniform(0.6, 1.0))))
         for i, v in enumerate(chops(nr, nth, nx))]
    more = {}
    if kind == "roundtrip" and nr >= 64 and rng.random() < 0.4:
        more["split"] = 6
    if kind in ("ab2", "etd"):
        more["steps"] = rng.choice([1, 2, 5, 10]) if nr * nth * nx <= 96 * 64 * 64 else 1
    return _case(kind, nr, nth, nx, c[0], c[1], c[2], **more)


# ------------------------------------------------------------------ inputs

def _config(case, seed=1234):
    """The configured physics of the case's scheme on its grid."""
    base = CONFIGS["etd_192x128x256" if case["kind"] == "etd" else
                   "grad_96x64x64" if case["kind"] == "vjp" else "ab2_64x32x32"]
    d = dict(base.__dict__)
    d.update(name="perf", seed=int(seed), notes=[], nr=case["nr"], nth=case["nth"], nx=case["nx"],
             nrchop=case["nrchop"], ntchop=case["ntchop"], nxchop=case["nxchop"])
    return Config(**d)


def _dims(case):
    """(m, n, k) extents of an FFF field."""
    return (min(case["ntchop"], case["nth"]), min(case["nrchop"] + 6, case["nr"]), 2 * case["nxchop"] - 1)


def _kept(case, pad=0):
    """Mask [m][n][1] of the radial modes below NRCHOP + pad - m."""
    nt, nn, _ = _dims(case)
    m = torch.arange(nt, device="cuda")[:, None, None]
    n = torch.arange(nn, device="cuda")[None, :, None]
    return n < case["nrchop"] + pad - m


def _axial(case):
    """Signed axial mode numbers in storage order."""
    nk = 2 * case["nxchop"] - 1
    k = torch.arange(nk, device="cuda", dtype=torch.float64)
    return torch.where(k < case["nxchop"], k, k - nk)


def _spectrum(case, gen, potential=False, decay=10.0):
    """Random FFF coefficients of a smooth real field: exp(-(n + m + |k|)/decay)
    times Gaussian, real at m = 0, chopped; `potential` divides by the
    horizontal Laplacian's eigenvalue and takes the value at infinity off."""
    nt, nn, nk = _dims(case)
    m = torch.arange(nt, device="cuda", dtype=torch.float64)[:, None, None]
    n = torch.arange(nn, device="cuda", dtype=torch.float64)[None, :, None]
    k = _axial(case)
    e = torch.randn(nt, nn, nk, dtype=torch.complex128, device="cuda", generator=gen)
    e = e * torch.exp(-(n + m + k.abs()) / decay) * _kept(case)
    back = torch.cat([torch.zeros(1, dtype=torch.long), torch.arange(nk - 1, 0, -1)]).cuda()
    e[0] = 0.5 * (e[0] + e[0][:, back].conj())
    if potential:
        deg = (m + n) * (m + n + 1)
        e = torch.where(deg > 0, e / deg.clamp(min=1.0), 0.0)
        at1 = torch.sqrt((2 * n[0] + 1) / 2)
        e[0, 0] = e[0, 0] - (at1 * e[0]).sum(0) / at1[0]
    return e.contiguous()


def _inputs(case, seed):
    """The input tensors of a case, from the seed alone: ([fields], [LN])."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    kind = case["kind"]
    if kind == "roundtrip":
        return [_spectrum(case, gen)], [0.0]
    if kind in ("rhs", "operators"):
        return [_spectrum(case, gen, potential=True) for _ in range(3)], [-0.5, 0.0, 0.0]
    if kind == "solves":
        return [_spectrum(case, gen) for _ in range(3)], [0.0, 0.0, 0.25]
    if kind == "project":  # r u_r, r u_phi, u_z samples of a smooth vector field, [r][z][packed theta]
        nr, nth, nx = case["nr"], case["nth"], case["nx"]
        x = torch.from_numpy(np.polynomial.legendre.leggauss(nr)[0]).cuda()[:, None, None]
        th = torch.arange(2 * nth, device="cuda", dtype=torch.float64)[None, None, :] * (math.pi / nth)
        z = torch.arange(nx, device="cuda", dtype=torch.float64)[None, :, None] * (2 * math.pi / nx)
        out = []
        for q in range(3):
            a = torch.rand(4, 3, dtype=torch.float64, device="cuda", generator=gen)
            f = 0.0
            for m in range(4):
                shape = (1 - x * x) ** (1 + (q < 2)) * torch.exp(-2.0 * a[m, 0] * (x + 0.3) ** 2)
                f = f + shape * torch.cos(m * th + 6 * a[m, 1]) * torch.cos((m % 3) * z + 6 * a[m, 2])
            out.append(torch.view_as_complex(f.reshape(nr, nx, nth, 2)).contiguous())
        return out, [0.0, 0.0, 0.0]
    raise ValueError(kind)


class _State:
    pass


def _take(s):
    """The result fields and their log terms, into the state's tensors."""
    for q, f in enumerate(s.result):
        s.ctx.DEVICE_COPY(f, False, M.FFF, s.out[q].data_ptr(), s.ln.data_ptr() + 8 * q)
    return {"fields": s.out, "ln": s.ln}


ALP = 2.0e6   # 2 / (NU DT) of the IVP configuration


def prepare(case, seed):
    s = _State()
    s.kind = kind = case["kind"]
    s.steps = int(case.get("steps", 1))
    if kind == "ensemble":
        cfgs = ensemble_configs(int(case["runs"]), int(case["grids"]))
        for i, c in enumerate(cfgs):
            c.seed = int(seed) % (1 << 28) + 7 * i
        s.ens = M.Ensemble(cfgs)
        s.states = []
        for ctx in s.ens.contexts:
            st = M.initial_state(ctx)
            ctx.initialize(*st)
            s.states.append(st)
        s.ens.step(2, graph=True)  # tunes and captures
        s.out = [[torch.zeros(ctx.NTCHOPDIM, ctx.NRCHOPDIM, ctx.NXCHOPDIM, dtype=torch.complex128, device="cuda")
                  for _ in range(3)] for ctx in s.ens.contexts]
        s.ens.sync()
        torch.cuda.synchronize()
        return s
    split = int(case.get("split", 0))
    s.ctx = ctx = M.Context(_config(case, int(seed) % (1 << 28)), precision=M.PREC_SPLIT if split else M.PREC_FP64,
                            split_slices=split)
    shape = _dims(case)
    if kind in ("ab2", "etd"):
        s.result = list(M.initial_state(ctx))
        ctx.initialize(*s.result)
        ctx.step(1, graph=True)  # captures the step
    elif kind == "vjp":
        s.solver = DeviceAB2(ctx)
        gen = torch.Generator(device="cuda").manual_seed(int(seed))
        s.x = tuple(_spectrum(case, gen, potential=True) for _ in range(6))
        s.x += (torch.tensor([-0.5, 0.0, 0.0, 0.0, 0.0, 0.0], dtype=torch.float64, device="cuda"),)
        s.bar = tuple(_spectrum(case, gen) for _ in range(6))
        s.bar += (torch.randn(6, dtype=torch.float64, device="cuda", generator=gen),)
        for _ in range(3):
            s.solver.step_vjp(s.x, s.bar)  # set-up, capture, replay
    else:
        tensors, lns = _inputs(case, seed)
        torch.cuda.synchronize()
        space = M.PPP if kind == "project" else M.FFF
        s.given = [ctx.field(space) for _ in tensors]
        ln = torch.tensor(lns, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        for q, (f, t) in enumerate(zip(s.given, tensors)):
            ctx.DEVICE_COPY(f, True, space, t.data_ptr(), ln.data_ptr() + 8 * q)
        ctx.sync()
        n = {"roundtrip": 1, "rhs": 3, "project": 2, "operators": 9, "solves": 3}[kind]
        s.result = [ctx.field(M.FFF) for _ in range(n)]
        if kind == "project":
            s.work = [ctx.field(M.PPP) for _ in range(3)]
    if kind != "vjp":
        s.out = [torch.zeros(shape, dtype=torch.complex128, device="cuda") for _ in s.result]
        s.ln = torch.zeros(len(s.result), dtype=torch.float64, device="cuda")
    ctx.sync()
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------ one pass

def run(s):
    if s.kind == "ensemble":
        s.ens.step(s.steps, graph=True)
        s.ens.sync()
        for ctx, fields, out in zip(s.ens.contexts, s.states, s.out):
            for f, t in zip(fields, out):
                ctx.DEVICE_COPY(f, False, M.FFF, t.data_ptr())
        return s.out
    ctx = s.ctx
    if s.kind == "roundtrip":
        f = s.result[0]
        ctx.COPY(f, s.given[0])
        ctx.TOFP(f)
        ctx.TOFF(f)
    elif s.kind == "rhs":
        ctx.CALC_BOUSSI_FORCE(*s.given, *s.result)
    elif s.kind == "project":
        for w, f in zip(s.work, s.given):
            ctx.COPY(w, f)
        ctx.PROJECT(*s.work, *s.result, LN=0.0)
    elif s.kind == "operators":
        psi, chi, b = s.given
        ctx.PC2VEL(psi, chi, *s.result[0:3])
        ctx.PC2VOR(psi, chi, *s.result[3:6])
        ctx.GRAD(b, *s.result[6:9])
    elif s.kind == "solves":
        ctx.IDEL2LN(s.given[0], s.result[0])
        ctx.IDEL2(s.given[1], s.result[1])
        ctx.IHELM(s.given[2], s.result[2], ALP)
    elif s.kind in ("ab2", "etd"):
        ctx.step(s.steps, graph=True)
    else:
        return list(s.solver.step_vjp(s.x, s.bar))
    return _take(s)


# ------------------------------------------------------------------ the work

def _sizes(case):
    nt, nn, nk = _dims(case)
    rows = sum(max(case["nrchop"] - m, 0) for m in range(nt))
    fff = 16.0 * nt * nn * nk
    gemm = 4.0 * case["nr"] * rows * nk                 # even/odd halves: 2 (NR/2) rows per real column
    ver = 5.0 * case["nr"] * nt * case["nx"] * math.log2(case["nx"])
    hor = 2.5 * case["nr"] * case["nx"] * 2 * case["nth"] * math.log2(2 * case["nth"])
    return fff, rows * nk * 2.0, gemm / 2, ver, hor


def work(case):
    """Each input read and each output written once; the arithmetic of the
    Legendre products (with the even/odd fold), the FFTs and the solves."""
    if case["kind"] == "ensemble":
        got = [work(_case("ab2", c.nr, c.nth, c.nx, c.nrchop, c.ntchop, c.nxchop, steps=case["steps"]))
               for c in ensemble_configs(int(case["runs"]), int(case["grids"]))]
        return {k: float(sum(g[k] for g in got)) for k in ("bytes", "flops")}
    fff, coef, gemm, ver, hor = _sizes(case)
    ppp = 16.0 * case["nr"] * case["nth"] * case["nx"]
    trans = gemm + ver + hor
    steps = int(case.get("steps", 1))
    kind = case["kind"]
    if kind == "roundtrip":
        return {"bytes": 2 * fff, "flops": 2 * trans}
    if kind == "rhs":
        return {"bytes": 6 * fff, "flops": 14 * (ver + hor) + 16 * gemm + 100 * coef}
    if kind == "project":
        return {"bytes": 3 * ppp + 2 * fff, "flops": 3 * (ver + hor) + 5 * gemm}
    if kind == "operators":
        return {"bytes": 12 * fff, "flops": 90 * coef}
    if kind == "solves":
        return {"bytes": 6 * fff, "flops": 3 * 14 * coef}
    if kind == "ab2":  # state and history in and out
        return {"bytes": steps * 12 * fff, "flops": steps * (14 * (ver + hor) + 16 * gemm + 250 * coef)}
    if kind == "etd":
        return {"bytes": steps * 20 * fff, "flops": steps * (13 * (ver + hor) + 18 * gemm + 350 * coef)}
    return {"bytes": 18 * fff, "flops": 2.5 * (14 * (ver + hor) + 16 * gemm + 250 * coef)}


# ------------------------------------------------------------------ plain 64-bit values

class _Plain:
    """The same maps in plain torch, in 64 bits: dense Legendre tables and band
    matrices, torch's FFTs and dense solves (ELL = 1, axial length 2 pi)."""

    def __init__(self, case):
        self.case = case
        self.nr, self.nth, self.nx, self.nxc = case["nr"], case["nth"], case["nx"], case["nxchop"]
        self.nrc = case["nrchop"]
        self.nt, self.nn, self.nk = _dims(case)
        x, w = np.polynomial.legendre.leggauss(self.nr)
        ne = self.nn + 4
        n = np.arange(ne)
        P = np.zeros((self.nt, self.nr, ne))
        xl = x.astype(np.longdouble)
        for m in range(self.nt):
            c = np.longdouble(0.5)
            for j in range(1, m + 1):
                c = c * np.longdouble(2 * j + 1) / np.longdouble(2 * j)
            v = np.zeros((self.nr, ne), dtype=np.longdouble)
            v[:, 0] = (-1) ** m * np.sqrt(c) * np.power(1 - xl * xl, np.longdouble(m) / 2)
            v[:, 1] = xl * np.sqrt(np.longdouble(2 * m + 3)) * v[:, 0]
            for q in range(2, ne):
                d = m + q
                a = np.sqrt(np.longdouble(4 * d * d - 1) / np.longdouble(d * d - m * m))
                b = np.sqrt(np.longdouble((d - 1) ** 2 - m * m) * np.longdouble(2 * d + 1)
                            / np.longdouble(d * d - m * m) / np.longdouble(2 * d - 3))
                v[:, q] = a * xl * v[:, q - 1] - b * v[:, q - 2]
            P[m] = v
        cuda = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).cuda()  # noqa: E731
        self.P, self.x, self.w = cuda(P), cuda(x), cuda(w)
        self.m = torch.arange(self.nt, device="cuda", dtype=torch.float64)[:, None, None]
        self.k = _axial(case)[None, None, :]
        self.norm0 = cuda(np.sqrt((2 * n + 1) / 2.0))
        # band matrices over ne rows: (1 - x), (1 - x^2) d/dx, the horizontal Laplacian
        XM, XX, D2 = (np.zeros((self.nt, ne, ne)) for _ in range(3))
        for m in range(self.nt):
            N = m + n.astype(np.float64)
            lo = np.sqrt((2 * N - 1).clip(1) / (2 * N + 1) * (N + m) / np.maximum(N - m, 1))  # norm(n-1)/norm(n)
            for q in range(ne):
                d = N[q]
                XM[m, q, q] = 1.0
                D2[m, q, q] = -2 * d * (d + 1) * (3 * d * d + 3 * d - m * m - 2) / (2 * d - 1) / (2 * d + 3)
                if q >= 1:
                    XM[m, q, q - 1] = -(d - m) / (2 * d - 1) * lo[q]
                    XX[m, q, q - 1] = -(d - 1) * (d - m) / (2 * d - 1) * lo[q]
                    D2[m, q, q - 1] = 2 * d * (d - m) * (d - 1) / (2 * d - 1) * lo[q]
                if q >= 2:
                    D2[m, q, q - 2] = (-(d - m - 1) * (d - m) * (d - 2) * (d - 1) / (2 * d - 3) / (2 * d - 1)
                                       * lo[q] * lo[q - 1])
                if q + 1 < ne:
                    XM[m, q, q + 1] = -(d + m + 1) / (2 * d + 3) / lo[q + 1]
                    XX[m, q, q + 1] = (d + 2) * (d + m + 1) / (2 * d + 3) / lo[q + 1]
                    D2[m, q, q + 1] = 2 * (d + 1) * (d + m + 1) * (d + 2) / (2 * d + 3) / lo[q + 1]
                if q + 2 < ne:
                    D2[m, q, q + 2] = (-(d + m + 1) * (d + m + 2) * (d + 3) * (d + 2) / (2 * d + 3) / (2 * d + 5)
                                       / lo[q + 1] / lo[q + 2])
        self.XM, self.XX, self.D2 = cuda(XM), cuda(XX), cuda(D2)

    def chop(self, a, pad):
        return a * _kept(self.case, pad)

    @staticmethod
    def mul(A, x):
        """Real matrices [m][i][j] times complex columns [m][j][k]."""
        y = torch.bmm(A.contiguous(), torch.view_as_real(x.contiguous()).flatten(2))
        return torch.view_as_complex(y.reshape(*y.shape[:2], -1, 2).contiguous())

    def band(self, B, a, pad):
        return self.chop(self.mul(B[:, :self.nn, :self.nn], self.chop(a, pad)), pad)

    def xxdx(self, a, ln, pad):
        b = self.band(self.XX, a, pad)
        b[0, 0, 0] += ln / self.norm0[0]
        b[0, 1, 0] += ln / self.norm0[1]
        return b

    def del2(self, a, ln, pad):
        b = self.band(self.D2, a, pad) - self.k ** 2 * self.chop(a, pad)
        for q, v in enumerate((4.0 / 3, -2.0, 2.0 / 3)):
            b[0, q, 0] += v * ln / self.norm0[q]
        return b

    def delsqh(self, a, ln, pad):
        n = self.m + torch.arange(self.nn, device="cuda")[None, :, None]
        b = -self.chop(a, pad) * n * (n + 1)
        b[0, 0, 0] = ln / self.norm0[0]
        return b

    def axial(self, a, ln, pad):
        return -self.band(self.XM, self.band(self.XM, self.delsqh(a, ln, pad), pad), pad)

    def grad(self, a, ln, pad):
        return [self.xxdx(a, ln, pad), self.chop(1j * self.m * a, pad), self.chop(1j * self.k * a, pad)]

    def pc2vel(self, p, lp, c, lc, pad):
        return [self.chop(1j * self.m * p, pad) + 1j * self.k * self.xxdx(c, lc, pad),
                -self.xxdx(p, lp, pad) - self.chop(self.m * self.k * c, pad), self.axial(c, lc, pad)]

    def pc2vor(self, p, lp, c, lc, pad):
        d = self.del2(c, lc, pad)
        return [-1j * self.m * self.chop(d, pad) + 1j * self.k * self.xxdx(p, lp, pad),
                self.xxdx(d, 0.0, pad) - self.chop(self.m * self.k * p, pad), self.axial(p, lp, pad)]

    def samples(self, a, pad):
        """Real samples [r][z][theta] of FFF coefficients."""
        f = self.mul(self.P[:, :, :self.nn], self.chop(a, pad))
        z = torch.zeros(self.nt, self.nr, self.nx, dtype=torch.complex128, device="cuda")
        z[:, :, :self.nxc] = f[:, :, :self.nxc]
        if self.nxc > 1:
            z[:, :, self.nx - self.nxc + 1:] = f[:, :, self.nxc:]
        z = torch.fft.ifft(z, dim=2) * self.nx
        z[0] = z[0].real.to(z.dtype)
        return torch.fft.irfft(z.permute(1, 2, 0), n=2 * self.nth, dim=2) * (2 * self.nth)

    def radial(self, f):
        """PFF [m][r][k] of real samples [r][z][theta]."""
        z = (torch.fft.rfft(f, dim=2) / (2 * self.nth))[:, :, :self.nt].permute(2, 0, 1).contiguous()
        z[0] = z[0].real.to(z.dtype)
        z = torch.fft.fft(z, dim=2) / self.nx
        return torch.cat([z[:, :, :self.nxc], z[:, :, self.nx - self.nxc + 1:]], dim=2) if self.nxc > 1 else z[:, :, :1]

    def spectral(self, F, pad):
        b = self.mul((self.P[:, :, :self.nn] * self.w[None, :, None]).transpose(1, 2), F)
        return self.chop(b, pad)

    def infinity(self, a, pad):
        """The m = 0 value at infinity taken off."""
        at1 = (self.norm0[:self.nn, None] * _kept(self.case, pad)[0]).to(a.dtype)
        a[0, 0] = a[0, 0] - (at1 * a[0]).sum(0) / self.norm0[0]
        return a

    def project(self, ur, up, uz):
        """(psi, del^2 chi) of a velocity form given as PFF, with LN = 0."""
        line = up[0, :, 0]
        c = (self.P[0, :, :self.nrc] * self.w[:, None]).transpose(0, 1).to(line.dtype) @ line
        ln = -(c.real * self.norm0[:self.nrc]).sum() / 2
        up = up.clone()
        up[0, :, 0] += ln * (1 + self.x)
        n = (self.m + torch.arange(self.nn, device="cuda")[None, :, None]).clamp(min=1.0)
        f = (self.w / (1 - self.x ** 2))[None, None, :]
        V = self.P[:, :, :self.nn].transpose(1, 2) / (n * (n + 1)) * f
        dP = torch.bmm(self.P, self.XX)[:, :, :self.nn]  # (1 - x^2) dP/dx
        D = dP.transpose(1, 2) / (n * (n + 1)) * f
        T = self.P[:, :, :self.nn].transpose(1, 2) * self.w[None, None, :]
        psi = self.chop(-1j * self.m * self.mul(V, ur) - self.mul(D, up), 0)
        w = self.chop(1j * self.k * self.mul(D, ur) + self.m * self.k * self.mul(V, up) - self.mul(T, uz), 0)
        return self.infinity(psi, 0), w

    def solve_m(self, a, b, alp, first):
        for m in range(first, self.nt):
            nn = max(self.nrc - m, 0)
            if nn:
                eye = torch.eye(nn, dtype=torch.float64, device="cuda")
                A = self.D2[m, :nn, :nn] - (self.k[0, 0] ** 2 + alp)[:, None, None] * eye
                y = torch.linalg.solve(A, torch.view_as_real(b[m, :nn].transpose(0, 1).contiguous()))
                a[m, :nn] = torch.view_as_complex(y.contiguous()).transpose(0, 1)
        return a

    def m0(self, A, b):
        y = torch.linalg.solve(A, torch.view_as_real(b.transpose(0, 1).contiguous()))
        return torch.view_as_complex(y.contiguous()).transpose(0, 1)

    def idel2ln(self, b):
        a, nn = torch.zeros_like(b), self.nrc
        b = self.chop(b, 0)
        A = self.D2[0, :nn, :nn] - (self.k[0, 0] ** 2)[:, None, None] * torch.eye(nn, dtype=torch.float64, device="cuda")
        for q, v in enumerate((4.0 / 3, -2.0, 2.0 / 3)):
            A[0, q, 0] += v * self.norm0[0] / self.norm0[q]
        a[0, :nn] = self.m0(A, b[0, :nn])
        ln = a[0, 0, 0].real * self.norm0[0]
        a[0, 0, 0] = 0
        return self.infinity(self.solve_m(a, b, 0.0, 1), 0), ln

    def idel2(self, b):
        """The LN argument absent: the (0, 0) mean is not solved for."""
        a, nn = torch.zeros_like(b), self.nrc
        b = self.chop(b, 0)
        A = self.D2[0, :nn, :nn] - (self.k[0, 0] ** 2)[:, None, None] * torch.eye(nn, dtype=torch.float64, device="cuda")
        for q, v in enumerate((4.0 / 3, -2.0, 2.0 / 3)):
            A[0, q, 0] += v * self.norm0[0] / self.norm0[q]
        A[0, 1:] = A[0, :-1].clone()
        A[0, 0] = 0.0
        A[0, 0, 0] = 1.0
        rhs = b[0, :nn].clone()
        rhs[1:, 0] = b[0, :nn - 1, 0]
        rhs[0, 0] = 0.0
        a[0, :nn] = self.m0(A, rhs)
        return self.infinity(self.solve_m(a, b, 0.0, 1), 0)

    def ihelm(self, b, lnb, alp):
        a, nn = torch.zeros_like(b), self.nrc
        b = self.chop(b, 0)
        ln = -lnb / alp
        for q, v in enumerate((4.0 / 3, -2.0, 2.0 / 3)):
            b[0, q, 0] -= v * ln / self.norm0[q]
        H = self.D2[0] - (self.k[0, 0] ** 2 + alp)[:, None, None] * torch.eye(self.D2.shape[1], dtype=torch.float64, device="cuda")
        A = (H[:, :nn + 1, :nn + 1] @ self.XM[0, :nn + 1, :nn + 1])[:, :nn - 1, :nn - 1]
        y = torch.zeros_like(b[0, :nn])
        y[:nn - 1] = self.m0(A, b[0, :nn - 1])
        a[0, :nn] = self.XM[0, :nn, :nn].to(y.dtype) @ y
        return self.chop(self.solve_m(a, b, alp, 1), 0), ln

    def force(self, p, c, b, ln, omega, bv0):
        g = [self.samples(f, 3) for f in self.grad(b, 0.0, 3)]
        u = [self.samples(f, 3) for f in self.pc2vel(p, ln[0], c, ln[1], 3)]
        o = [self.samples(f, 3) for f in self.pc2vor(p, ln[0], c, ln[1], 3)]
        bs = self.samples(b, 0)
        r2 = ((1 + self.x) / (1 - self.x))[:, None, None]
        n1 = u[1] * o[2] - u[2] * o[1] + 2 * omega * u[1]
        n2 = u[2] * o[0] - u[0] * o[2] - 2 * omega * u[0]
        n3 = (u[0] * o[1] - u[1] * o[0]) / r2 - bs
        nb = -((u[0] * g[0] + u[1] * g[1]) / r2 + u[2] * g[2]) + bv0 ** 2 * u[2]
        psi, w = self.project(*[self.radial(f) for f in (n1, n2, n3)])
        chi, lc = self.idel2ln(w)
        return [psi, chi, self.spectral(self.radial(nb), 0)], torch.stack([torch.zeros_like(lc), lc, torch.zeros_like(lc)])


def exact(case, seed):
    kind = case["kind"]
    if kind in ("ab2", "etd", "vjp", "ensemble"):
        return None  # whole steps: their parts are the other cases
    fields, ln = _inputs(case, seed)
    if kind == "roundtrip":  # the transforms invert one another on chopped fields
        return {"fields": fields, "ln": torch.zeros(1, dtype=torch.float64)}
    p = _Plain(case)
    zeros = lambda n: torch.zeros(n, dtype=torch.float64)  # noqa: E731
    if kind == "rhs":
        cfg = _config(case)
        f, lns = p.force(*fields, ln, cfg.omega, cfg.bv0)
        return {"fields": f, "ln": lns}
    if kind == "project":
        f = p.project(*[p.radial(torch.view_as_real(t).flatten(2)) for t in fields])
        return {"fields": list(f), "ln": zeros(2)}
    if kind == "operators":
        f = p.pc2vel(fields[0], ln[0], fields[1], ln[1], 0) + p.pc2vor(fields[0], ln[0], fields[1], ln[1], 0)
        return {"fields": f + p.grad(fields[2], ln[2], 0), "ln": zeros(9)}
    a0, l0 = p.idel2ln(fields[0])
    a2, l2 = p.ihelm(fields[2], ln[2], ALP)
    return {"fields": [a0, p.idel2(fields[1]), a2], "ln": torch.tensor([float(l0), 0.0, l2], dtype=torch.float64)}
