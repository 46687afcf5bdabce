"""The work a user has this framework do, as cases that can be timed and compared: matvecs on device buffers, solves,
adjoint gradients and scattered fields, through the Python front end and the C ABI it binds.

A case is a dict:
  kind    "matvec" (adda_gb300_matvec_device), "solve" (Context.solve_device + cross sections), "vjp"
          (Context.vjp_chi) or "fields" (Context.scattered_fields + cross sections)
  shape, grid, ry, rz   the particle: A.make_particle(shape, grid, (ry, rz)); the FFT grid is the reference's fftFit
  rhs     right-hand sides in one call
  prec    "fp64" or "fp32" (matvec), "fp64" or "mixed" (solve, vjp)
  her     matvec with the Hermitian transpose (CGNR's other direction)
  dipole  every dipole has its own polarisability (inhomogeneous media), else one material
  surface the particle stands above a substrate (image relation)
  method, eps   Krylov method and relative residual of a solve
  dirs    scattering directions

exact() restates each result in complex128 with torch: the interaction as one zero-padded cyclic convolution, solves by
a plain BiCGStab on it, fields as a direct sum.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(ROOT, "a-dda_gb300") not in sys.path:
    sys.path.insert(0, os.path.join(ROOT, "a-dda_gb300"))
import adda_gb300 as A  # noqa: E402

M_REF, DPL = 1.33 + 0.01j, 15.0  # refractive index and dipoles per wavelength of the benchmark sphere
BASE = dict(shape="sphere", grid=16, ry=1.0, rz=1.0, rhs=2, prec="fp32", her=False, dipole=False, surface=False,
            method="qmr", eps=1e-10, dirs=0, m_re=M_REF.real, m_im=M_REF.imag, dpl=DPL)


def _case(name, kind, **kw):
    return dict(BASE, kind=kind, **dict(kw, **({"name": name} if name else {})))


def listed():
    return [
        # the smallest call: one polarisation of the 16^3 sphere (FFT grid 32^3); launches and latency count
        _case("mv32_sphere16_r1", "matvec", grid=16, rhs=1),
        # the plain FP64 method on the 16^3 sphere, m = 1.5, dpl 10, both polarisations, converged
        _case("solve64_sphere16", "solve", grid=16, prec="fp64", m_re=1.5, m_im=0.0, dpl=10.0),
        # the inhomogeneous 48^3 cube (grid 96^3), every dipole its own polarisability, Hermitian direction
        _case("mv32_cube48_dipole_her", "matvec", shape="box", grid=48, dipole=True, her=True),
        # an ellipsoid of the orientation batch: uneven grid 192 x 154 x 112, 8 right-hand sides
        _case("mv32_ell96_r8", "matvec", shape="ellipsoid", grid=96, ry=0.79, rz=0.583, rhs=8),
        # the benchmark sphere, 128^3 box, grid 256^3, both polarisations: the matvec of the mixed solver's iterations
        _case("mv32_sphere128", "matvec", grid=128),
        # the same in FP64: the matvec of the plain FP64 solver and of the refinement residual
        _case("mv64_sphere128", "matvec", grid=128, prec="fp64"),
        # the largest: 256^3 sphere, grid 512^3
        _case("mv32_sphere256", "matvec", grid=256),
        # a particle above a substrate: the reflected interaction in the same matvec
        _case("mv32_surf64", "matvec", grid=64, surface=True),
        # a whole mixed-precision solve, both polarisations, converged cross sections (grid 128^3)
        _case("solve_mixed_sphere64", "solve", grid=64, prec="mixed"),
        # a batch of orientations of an ellipsoid on an uneven grid, BiCGStab
        _case("solve_mixed_ell48_r8", "solve", shape="ellipsoid", grid=48, ry=0.8, rz=0.6, rhs=8, prec="mixed",
              method="bicgstab", m_re=1.4, m_im=0.02),
        # gradients of Cext and Cabs with respect to every dipole of an inhomogeneous cube: the adjoint solve
        _case("vjp_cube32", "vjp", shape="box", grid=32, dipole=True, prec="mixed"),
        # scattering amplitudes of a 64^3 sphere in the directions of the reference's default integration grid
        _case("fields_sphere64", "fields", grid=64, dirs=2080),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi):
    """a box size: even, as the reference's shapes have it"""
    return 2 * _log(rng, lo / 2, hi / 2)


def draw(rng):
    kind = rng.choice(["matvec", "matvec", "matvec", "solve", "vjp", "fields"])
    shape = rng.choice(["sphere", "ellipsoid", "box"])
    ry, rz = (1.0, 1.0) if shape == "sphere" else (round(rng.uniform(0.5, 1.0), 3), round(rng.uniform(0.5, 1.0), 3))
    kw = dict(shape=shape, ry=ry, rz=rz)
    if kind == "matvec":
        prec = rng.choice(["fp32", "fp32", "fp64"])
        hi = 200 if prec == "fp32" else 110
        grid = _box(rng, 10, hi)
        most = max(1, min(16, int(2 * (hi / grid) ** 3)))
        return _case(None, kind, grid=grid, prec=prec, rhs=min(most, rng.choice([1, 2, 2, 3, 4, 8, 16])),
                     her=rng.random() < 0.3, dipole=rng.random() < 0.3, surface=rng.random() < 0.2 and grid <= 100,
                     **kw)
    if kind == "solve":
        prec = rng.choice(["mixed", "mixed", "fp64"])
        hi = 64 if prec == "mixed" else 24
        grid = _box(rng, 8, hi)
        return _case(None, kind, grid=grid, prec=prec,
                     rhs=min(rng.choice([1, 2, 2, 4, 6]), int(2 * (hi / grid) ** 3)), method=rng.choice(["qmr", "bicgstab"]),
                     m_re=round(rng.uniform(1.2, 1.5), 3), m_im=round(rng.uniform(0.01, 0.05), 4), **kw)
    if kind == "vjp":
        return _case(None, kind, grid=_box(rng, 8, 40), dipole=rng.random() < 0.7, prec="mixed", **kw)
    grid = _box(rng, 12, 80)
    return _case(None, kind, grid=grid, rhs=rng.choice([1, 2, 4]),
                 dirs=_log(rng, 30, max(60, int(2080 * min(1.0, (64 / grid) ** 3)))), **kw)


# ---------------------------------------------------------------------------------------------------------------------
# inputs: lattice, polarisabilities, fields (host arrays and seeded vectors), shared by prepare and exact

class _Inputs:
    pass


def _inputs(c, seed):
    s = _Inputs()
    pars = None if c["shape"] == "sphere" else (c["ry"], c["rz"])
    s.box, s.pos, s.mat = A.make_particle(c["shape"], c["grid"], pars)
    s.n, s.R = len(s.pos), c["rhs"]
    s.grid = (A.fft_fit(2 * s.box[0]), A.fft_fit(2 * s.box[1]), A.fft_fit(2 * s.box[2], 2))
    s.k, s.kd = 1.0, 2 * math.pi / c["dpl"]
    s.gs = s.kd / s.k
    rng = np.random.default_rng(seed)
    m = complex(c["m_re"], c["m_im"])
    if c["dipole"]:
        m = rng.uniform(1.3, 1.7, s.n) + 1j * rng.uniform(0.0, 0.05, s.n)
    # Clausius-Mossotti with the radiative reaction correction
    a0 = s.gs ** 3 * 3 / (4 * np.pi) * (m * m - 1) / (m * m + 2)
    cc = 1 / (1 / a0 - 2j / 3 * s.k ** 3)
    s.cc = np.repeat(np.atleast_1d(cc).astype(np.complex128)[:, None], 3, axis=1)  # [nmat or n, 3]
    s.f = 4 * np.pi / s.gs ** 3 * -1 / ((m * m - 1) / (4 * np.pi)) ** 2 / (4 * np.pi) * np.ones(s.n)  # d(1/a)/dchi, CM
    s.surface = None
    if c["surface"]:  # the centre one box height above a substrate of index 1.5
        s.surface = dict(zsum_shift=2 * (s.box[2] - (s.box[2] - 1) / 2.0), msub=1.5 + 0j, relation="img")
    # incident frames: orientations about random axes, both polarisations of each
    s.prop, s.pol = np.zeros((s.R, 3)), np.zeros((s.R, 3))
    for r in range(s.R):
        if r % 2 == 0:
            q, t = np.linalg.qr(rng.standard_normal((3, 3)))
            q = q * np.sign(np.diag(t))
        s.prop[r], s.pol[r] = q[:, 0], q[:, 1 + r % 2]
    return s


def _context(c, s, rhs=None):
    ctx = A.Context(s.box, s.pos, s.mat, s.gs, s.k, s.grid, nrhs_max=rhs or s.R, surface=s.surface)
    ctx.init_dmatrix()
    for r in range(rhs or s.R):
        if c["dipole"]:
            ctx.set_cc_dipole(r, s.cc)
        else:
            ctx.set_cc(r, s.cc)
    return ctx


def _vectors(c, s, seed, dtype=torch.complex128):
    """seeded Krylov-like vectors [R, 3N] on the GPU"""
    g = torch.Generator("cuda").manual_seed(int(seed))
    return torch.randn((s.R, 3 * s.n), dtype=torch.complex64, device="cuda", generator=g).to(dtype)


def _waves(s):
    """incident plane waves pol * exp(i k r.prop) at the dipoles (r from the box centre), [R, 3N] on the GPU"""
    pos = torch.from_numpy(s.pos.astype(np.float64)).cuda() - (torch.tensor(s.box, dtype=torch.float64) - 1).cuda() / 2
    ph = s.kd * (torch.from_numpy(s.prop).cuda() @ pos.T)
    e = torch.exp(1j * ph)[:, :, None] * torch.from_numpy(s.pol).cuda()[:, None, :]
    return e.reshape(s.R, 3 * s.n).contiguous()


def _dirs(c, seed):
    d = np.random.default_rng(seed + 1).standard_normal((c["dirs"], 3))
    return d / np.linalg.norm(d, axis=1, keepdims=True)


def prepare(case, seed):
    s = _inputs(case, seed)
    st = dict(case=case, s=s, kind=case["kind"])
    if case["kind"] == "matvec":
        st["ctx"] = _context(case, s)
        st["x"] = _vectors(case, s, seed, torch.complex64 if case["prec"] == "fp32" else torch.complex128)
        st["y"] = torch.empty_like(st["x"])
        st["args"] = (st["ctx"].h, A.PREC[case["prec"]], s.R, ctypes.c_void_p(st["x"].data_ptr()),
                      ctypes.c_void_p(st["y"].data_ptr()), None, int(case["her"]))
    elif case["kind"] == "solve":
        st["ctx"] = _context(case, s)
        st["e"] = _waves(s)
        st["x"], st["p"] = torch.empty_like(st["e"]), torch.empty_like(st["e"])
    elif case["kind"] == "vjp":
        # the forward solution stays in the context, as after a user's forward pass
        st["ctx"] = _context(case, s, 2)
        e = _waves(s)
        st["ctx"].solve_device(e.data_ptr(), s.R, prec="fp64", eps=1e-11)
    else:
        # polarisations of a solution the context holds: x handed over as the starting vector, no iterations
        st["ctx"] = _context(case, s)
        x, e = _vectors(case, s, seed), _waves(s)
        st["ctx"].solve_device(e.data_ptr(), s.R, x.data_ptr(), prec="fp64", maxiter=0, init="x0")
        st["dirs"] = _dirs(case, seed)
    torch.cuda.synchronize()
    return st


def run(st):
    c, ctx, s = st["case"], st["ctx"], st["s"]
    if st["kind"] == "matvec":
        if ctx.L.adda_gb300_matvec_device(*st["args"]):
            raise RuntimeError(ctx.L.adda_gb300_last_error().decode())
        return st["y"]
    if st["kind"] == "solve":
        ctx.solve_device(st["e"].data_ptr(), s.R, st["x"].data_ptr(), st["p"].data_ptr(), method=c["method"],
                         prec=c["prec"], eps=c["eps"])
        return dict(x=st["x"], p=st["p"], cross=ctx.cross_sections(s.prop, s.pol))
    if st["kind"] == "vjp":
        return ctx.vjp_chi(0, s.prop[0], s.pol[0], s.f, method=c["method"], prec=c["prec"], eps=1e-11)
    return dict(e=ctx.scattered_fields(st["dirs"], s.R), cross=ctx.cross_sections(s.prop, s.pol))


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without

def work(case):
    pars = None if case["shape"] == "sphere" else (case["ry"], case["rz"])
    box, pos, _ = A.make_particle(case["shape"], case["grid"], pars)
    n, R = len(pos), case["rhs"]
    g = (A.fft_fit(2 * box[0]), A.fft_fit(2 * box[1]), A.fft_fit(2 * box[2], 2))
    if case["kind"] == "fields":
        nd = case["dirs"]
        return dict(bytes=R * n * 48 + R * nd * 48, flops=24.0 * n * R * nd)
    size = 16 if case["prec"] == "fp64" else 8
    dbytes = 6 * size * g[0] * (g[1] // 2 + 1) * (g[2] // 2 + 1)
    if case["surface"]:
        dbytes += 6 * size * g[0] * (g[1] // 2 + 1) * g[2]
    cells = g[0] * g[1] * g[2]
    # forward and inverse transforms of three components, the zero-padded lines skipped, and the 3x3 products
    lines = 5.0 * (box[1] * box[2] * g[0] * math.log2(g[0]) + box[1] * g[0] * g[2] * math.log2(g[2])
                   + cells * math.log2(g[1]))
    flops = R * (6 * lines + 72.0 * cells) * (1.6 if case["surface"] else 1.0)
    vec = 3 * n * R * size
    cc = 3 * n * size * (R if case["dipole"] else 0)
    if case["kind"] == "matvec":
        return dict(bytes=2 * vec + dbytes + cc + 4 * n, flops=flops)
    # an iterative solve: about 40 matvecs of these, each with ten passes over vectors of 16 bytes an element
    its = 40
    R2 = 2 if case["kind"] == "vjp" else R
    return dict(bytes=its * (dbytes + cc + R2 * 3 * n * (2 * size + 160)), flops=its * flops * R2 / R)


# ---------------------------------------------------------------------------------------------------------------------
# the same results in 64 bits, in plain torch

class _Exact:
    """A = I - S (G + GR) S on the dipoles, the sums over dipoles as cyclic convolutions of twice the box (per axis)"""

    def __init__(self, c, s):
        self.s = s
        b = s.box
        self.g = tuple(2 * v for v in b)
        pos = torch.from_numpy(s.pos.astype(np.int64)).cuda()
        self.idx = (pos[:, 2] * self.g[1] + pos[:, 1]) * self.g[0] + pos[:, 0]
        self.idr = ((b[2] - 1 - pos[:, 2]) * self.g[1] + pos[:, 1]) * self.g[0] + pos[:, 0]  # heights reversed
        cc = torch.from_numpy(s.cc).cuda()
        self.cc = cc if len(cc) == s.n else cc.expand(s.n, 3)
        self.S = torch.sqrt(self.cc)
        ax = [torch.arange(v, dtype=torch.float64, device="cuda") for v in self.g]
        off = [torch.where(a < w, a, a - 2 * w) for a, w in zip(ax, b)]
        self.G = self._tensor(off[0], off[1], off[2], None)
        self.GR = None
        if s.surface:
            self.GR = self._tensor(off[0], off[1], off[2] + (b[2] - 1) + s.surface["zsum_shift"], s.surface["msub"])

    def _tensor(self, x, y, z, msub):
        """FFT of the point-dipole tensor (xx, xy, xz, yy, yz, zz) at lattice offsets; msub: the image-dipole one"""
        s = self.s
        Z, Y, X = torch.meshgrid(z, y, x, indexing="ij")
        r = torch.sqrt(X * X + Y * Y + Z * Z)
        zero = r == 0
        r[zero] = 1.0
        q = [X / r, Y / r, Z / r]
        kr = s.k * s.gs * r
        e = torch.exp(1j * kr) / (s.gs * r) ** 3
        e[zero] = 0
        del X, Y, Z, r
        if msub is not None:
            e = e * ((1 - msub ** 2) / (1 + msub ** 2))
        out = []
        for a, b in ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2)):
            qq = q[a] * q[b]
            t = torch.complex((3 - kr * kr) * qq, -3 * kr * qq)
            if a == b:
                t = t + torch.complex(kr * kr - 1, kr)
            if msub is not None and 2 in (a, b):
                t = -t
            out.append(torch.fft.fftn(t * e))
        return out

    def _grid(self, v, idx):
        f = torch.zeros(self.g[2] * self.g[1] * self.g[0], dtype=torch.complex128, device="cuda")
        f[idx] = v
        return torch.fft.fftn(f.view(self.g[2], self.g[1], self.g[0]))

    def __call__(self, x, her=False):
        """A x of one vector [3N] (her: A^H x; A is complex symmetric)"""
        v = x.view(-1, 3)
        v = v.conj() if her else v
        p = self.S * v
        G = self.G
        P = [self._grid(p[:, a], self.idx) for a in range(3)]
        F = [G[0] * P[0] + G[1] * P[1] + G[2] * P[2], G[1] * P[0] + G[3] * P[1] + G[4] * P[2],
             G[2] * P[0] + G[4] * P[1] + G[5] * P[2]]
        if self.GR:
            G = self.GR
            P = [self._grid(p[:, a], self.idr) for a in range(3)]
            F = [F[0] + G[0] * P[0] + G[1] * P[1] + G[2] * P[2], F[1] + G[1] * P[0] + G[3] * P[1] + G[4] * P[2],
                 F[2] - G[2] * P[0] - G[4] * P[1] + G[5] * P[2]]
        E = torch.stack([torch.fft.ifftn(f).reshape(-1)[self.idx] for f in F], 1)
        y = v - self.S * E
        return (y.conj() if her else y).reshape(-1)

    def solve(self, b, eps=2e-14, most=4000):
        """BiCGStab, restarted from the true residual, to eps or to the level rounding allows"""
        x = torch.zeros_like(b)
        nb, best, xbest = torch.linalg.norm(b), math.inf, x
        for _ in range(6):
            r = b - self(x)
            res = float(torch.linalg.norm(r) / nb)
            if res < best:
                best, xbest = res, x.clone()
            if res < eps:
                break
            rt, p, rho = r.clone(), r.clone(), torch.vdot(r, r)
            for _ in range(most):
                v = self(p)
                al = rho / torch.vdot(rt, v)
                q = r - al * v
                t = self(q)
                om = torch.vdot(t, q) / torch.vdot(t, t)
                x = x + al * p + om * q
                r = q - om * t
                if float(torch.linalg.norm(r) / nb) < 0.3 * eps:
                    break
                rn = torch.vdot(rt, r)
                p = r + (rn / rho) * (al / om) * (p - om * v)
                rho = rn
        return xbest


def _cross(c, s, P, cc):
    """extinction (optical theorem) and absorption cross sections of polarisations P [R, N, 3]"""
    pos = torch.from_numpy(s.pos.astype(np.float64)).cuda() - (torch.tensor(s.box, dtype=torch.float64) - 1).cuda() / 2
    ce, ca = np.zeros(s.R), np.zeros(s.R)
    for r in range(s.R):
        n, e = torch.from_numpy(s.prop[r]).cuda(), torch.from_numpy(s.pol[r]).cuda()
        f = torch.exp(-1j * s.kd * (pos @ n)) @ P[r]
        f = f - n * (f @ n.to(f.dtype))
        ce[r] = float((-1j * s.k ** 3 * f @ e.to(f.dtype)).real) * 4 * math.pi / s.k ** 2
        mu = -(1 / cc).imag - 2 * s.k ** 3 / 3
        ca[r] = 4 * math.pi * s.k * float((mu * P[r].abs() ** 2).sum())
    return ce, ca


def exact(case, seed):
    s = _inputs(case, seed)
    if case["kind"] == "fields":
        cc = torch.from_numpy(s.cc).cuda().expand(s.n, 3)
        P = torch.sqrt(cc) * _vectors(case, s, seed).view(s.R, s.n, 3)
        pos = torch.from_numpy(s.pos.astype(np.float64)).cuda() - (torch.tensor(s.box, dtype=torch.float64) - 1).cuda() / 2
        d = torch.from_numpy(_dirs(case, seed)).cuda()
        out = torch.zeros((s.R, len(d), 3), dtype=torch.complex128, device="cuda")
        for i in range(0, len(d), 64):
            w = torch.exp(-1j * s.kd * (d[i:i + 64] @ pos.T))
            for r in range(s.R):
                f = w @ P[r]
                out[r, i:i + 64] = -1j * s.k ** 3 * (f - d[i:i + 64] * (f * d[i:i + 64]).sum(1, keepdim=True))
        return dict(e=out, cross=_cross(case, s, P, cc))
    A_ = _Exact(case, s)
    if case["kind"] == "matvec":
        x = _vectors(case, s, seed)
        return torch.stack([A_(x[r], case["her"]) for r in range(s.R)])
    e = _waves(s)
    b = [(A_.S * e[r].view(-1, 3)).reshape(-1) for r in range(s.R)]
    if case["kind"] == "solve":
        x = torch.stack([A_.solve(v) for v in b])
        p = A_.S * x.view(s.R, s.n, 3)
        return dict(x=x, p=p.reshape(s.R, -1), cross=_cross(case, s, p, A_.cc))
    # gradients: lambda from the extinction's adjoint source, nu from the absorption's
    P = A_.S * A_.solve(b[0]).view(-1, 3)
    pos = torch.from_numpy(s.pos.astype(np.float64)).cuda() - (torch.tensor(s.box, dtype=torch.float64) - 1).cuda() / 2
    w = -4j * math.pi * s.k * torch.exp(-1j * s.kd * (pos @ torch.from_numpy(s.prop[0]).cuda()))
    mu = -(1 / A_.cc).imag - 2 * s.k ** 3 / 3
    src = [w[:, None] * torch.from_numpy(s.pol[0]).cuda(), mu * P.conj()]
    lam, nu = [A_.S * A_.solve((A_.S * q).reshape(-1)).view(-1, 3) for q in src]
    f = torch.from_numpy(s.f.astype(np.complex128)).cuda()
    g = -f * (lam * P).sum(1)
    h = f * (nu * P).sum(1)
    p2 = (P.abs() ** 2).sum(1)
    ka = 4 * math.pi * s.k
    return (torch.stack([g.real, -g.imag], 1),
            torch.stack([ka * (-f.imag * p2 - 2 * h.real), ka * (-f.real * p2 + 2 * h.imag)], 1))
