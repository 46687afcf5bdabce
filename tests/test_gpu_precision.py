"""Results to FP64 rounding where one part of the data is much smaller than another, against sums in extended precision.

Matvec tolerance: a component of y = x + S.X carries the rounding of the last sum (2^-53) and the noise of six transforms of
up to 6 stages and of the D product, 2^-53 each and random, on S.X, which is below half of y here:
(1 + sqrt(6 * 6 + 1) / 2) * 2^-53 = 4.5e-16; twice that."""
import math

import numpy as np
import pytest

from test_gpu_parity import context, cube_setup, random_vec

pytestmark = pytest.mark.gpu
TOL = 9e-16
LD, CLD = np.longdouble, np.clongdouble


def matvec_direct(s, cc, x, pick=None):
    """x - S G S x by a direct sum over the dipoles in extended precision, [n, 3] or at the picked dipoles"""
    S = np.sqrt(cc.reshape(-1)[:3].astype(CLD))
    v = x * S
    pick = range(s.n) if pick is None else pick
    pos, out = s.pos.astype(LD), np.empty((len(pick), 3), CLD)
    kd = LD(s.wavenum) * LD(s.gridspace)
    for k, i in enumerate(pick):
        d = pos[i] - pos
        d[i] = 1
        r = np.sqrt((d * d).sum(1))
        q, kr = d / r[:, None], kd * r
        e = np.exp(1j * kr.astype(CLD)) / (LD(s.gridspace) * r) ** 3
        e[i] = 0
        a, b = e * (kr * kr - 1 + 1j * kr), e * (3 - kr * kr - 3j * kr) * (q * v).sum(1)
        out[k] = x[i] - S * (a[:, None] * v + b[:, None] * q).sum(0)
    return out


@pytest.mark.parametrize("box", [(16, 16, 1), (16, 1, 16), (1, 16, 16), (60, 1, 1), (1, 60, 1), (1, 1, 60), (1, 1, 1)])
def test_uncoupled_components_of_a_flat_box(box):
    """in a box one dipole thick along an axis that component couples to no other (in a row none couples): each keeps its
    own relative precision, whatever the others' size"""
    s = cube_setup(box, tuple(2 * b for b in box))
    free = [a for a in range(3) if box[a] == 1] if sum(b > 1 for b in box) == 2 else [0, 1, 2]
    c = context(s, R=6)
    for r in range(6):
        c.set_cc(r, s.cc[0].reshape(1, 3))
    scales = [[10.0 ** (-4 * ((a + k) % 3)) for a in range(3)] for k in range(3)]
    scales += [[10.0 ** (-9 * ((a + k) % 3)) for a in range(3)] for k in range(3)]
    x = random_vec(s.n, 6, sum(box)).reshape(6, s.n, 3) * np.array(scales)[:, None, :]
    y = c.matvec(x.reshape(6, -1), "fp64")[0].reshape(6, s.n, 3)
    for r in range(6):
        want = matvec_direct(s, s.cc[0], x[r])
        for a in free:
            err = np.sqrt(float((np.abs(y[r, :, a] - want[:, a]) ** 2).sum() / (np.abs(want[:, a]) ** 2).sum()))
            assert err < TOL, (r, a, err)
    c.close()


# ---------------------------------------------------------------------------------------------------------------------
# Scattered fields. Tolerance: three phase factors of a term and the box centre's have 1.5 * 2^-53 each (a sine's 1 ulp
# and its rounding to the table), the polarisations 2^-54 of their largest, about 5 times their rms, and the last sums, the
# projection and the products a handful of 2^-53; all random: sqrt(4 * 1.5^2 + 2.5^2 + 6) * 2^-53 = 5e-16 of the rms field,
# with a factor of 4 for the fields of single directions.
FIELD_TOL = 2e-15


def full_box(box, k, dpl=15.0):
    s = cube_setup(box, tuple(2 * b for b in box))
    s.kd, s.wavenum = 2 * math.pi / dpl, k
    s.gridspace = s.kd / k
    s.cc = [np.array([(0.3 + 0.02j) * s.gridspace ** 3] * 3)] * 2
    return s


def fields_of(s, x, dirs, among=4000):
    """the context's fields for x handed over as the solution (no iterations), among so many directions that they come
    from the tables (0: these alone), and the polarisations they are of"""
    import torch
    R, nd = len(x), len(dirs)
    dirs = np.concatenate([dirs, some_dirs(max(among - nd, 0), 99)])
    c = context(s, R=R)
    d_x = torch.from_numpy(np.ascontiguousarray(x.reshape(R, -1), dtype=np.complex128).view(np.float64)).cuda()
    d_p = torch.empty_like(d_x)
    torch.cuda.synchronize()
    c.solve_device(d_x.data_ptr(), R, d_x.data_ptr(), d_p.data_ptr(), prec="fp64", maxiter=0, init="x0")
    torch.cuda.synchronize()
    e = c.scattered_fields(dirs, R)[:, :nd]
    c.close()
    return e, d_p.cpu().numpy().view(np.complex128).reshape(R, s.n, 3)


def fields_direct(s, P, dirs):
    """-i k^3 (I - nn) sum P exp(-i k n.r), r from the box centre, in extended precision"""
    r = LD(s.gridspace) * (s.pos.astype(LD) - (np.array(s.box, dtype=LD) - 1) / 2)
    out = np.empty((len(P), len(dirs), 3), CLD)
    for i, d in enumerate(dirs.astype(LD)):
        w = np.exp(-1j * (LD(s.wavenum) * (r @ d)).astype(CLD))
        for q in range(len(P)):
            f = w @ P[q].astype(CLD)
            out[q, i] = -1j * LD(s.wavenum) ** 3 * (f - d * (f @ d))
    return out


def field_errors(got, want):
    """per RHS and direction, relative to that direction's field"""
    n = lambda v: np.sqrt((np.abs(v) ** 2).sum(-1).astype(np.float64))
    return n(got - want) / n(want)


def some_dirs(n, seed):
    d = np.random.default_rng(seed).standard_normal((n, 3))
    return d / np.linalg.norm(d, axis=1, keepdims=True)


@pytest.mark.parametrize("among", [0, 4000])
@pytest.mark.parametrize("k", [2 * math.pi, 2 * math.pi / 0.6328, 0.7, 9.3e6])
@pytest.mark.parametrize("box", [(300, 2, 3), (3, 300, 2), (2, 3, 300)])
def test_fields_with_any_wave_number(box, k, among):
    """k times the spacing is not a double: every factor of the phase, and the box centre's, takes the same value of it"""
    s = full_box(box, k)
    x = random_vec(s.n, 2, 7)
    dirs = np.concatenate([some_dirs(40, 3), [[0.8, 0.6, 0], [0.6, 0, 0.8]]])
    e, P = fields_of(s, x, dirs, among)
    err = field_errors(e, fields_direct(s, P, dirs))
    assert np.sqrt((err ** 2).mean()) < FIELD_TOL


@pytest.mark.parametrize("size", [1.0, 0.25, 0.0625])
@pytest.mark.parametrize("d", [(1, 0, 0), (-1, 0, 0), (0, 0.6, 0.8)])
def test_field_roundings_do_not_lean(size, d):
    """a plate's polarisations of random sign whose last bit falls in the middle of the fixed-point unit (one larger dipole
    sets the unit): if the middle always goes up, 40000 of them add 1e-16 each to a field of 200"""
    s = full_box((1, 200, 200), 1.0)
    s.cc = [np.ones(3)] * 2
    g = np.random.default_rng(5)
    v = size * (1 + 2.0 ** -52)
    x = v * (g.choice([-1, 1], (2, s.n, 3)) + 1j * g.choice([-1, 1], (2, s.n, 3)))
    x[:, 0] = 1
    e, P = fields_of(s, x, np.array([d], dtype=float))
    assert np.array_equal(P, x)
    assert field_errors(e, fields_direct(s, P, np.array([d], dtype=float))).max() < FIELD_TOL


@pytest.mark.parametrize("scale", [(1, 1e-3, 1e-6), (1e-6, 1, 1e-9), (1e-12, 1e-7, 1), (1, 1e-200, 1e-300)])
def test_fields_along_a_dominant_component(scale):
    """the field in the direction of a component is made of the other two alone, however small they are"""
    s = full_box((24, 18, 14), 1.0)
    x = random_vec(s.n, 6, 11).reshape(6, s.n, 3) * np.array(scale)
    dirs = np.concatenate([np.eye(3), -np.eye(3), some_dirs(10, 5)])
    e, P = fields_of(s, x, dirs)
    want = fields_direct(s, P, dirs)
    n = lambda v: np.sqrt((np.abs(v).astype(LD) ** 2).sum((0, 2)))  # per direction, over the right-hand sides
    assert (n(e - want) / n(want)).max() < FIELD_TOL


@pytest.mark.parametrize("shape,R,dirs", [((10, 9, 8), 1, (1, 2, 31, 33, 340, 360)), ((40, 30, 25), 2, (1, 2, 5, 6, 7)),
                                          ((1, 1, 1), 3, (1, 40))])
def test_fields_of_few_directions(shape, R, dirs):
    """both sides of the line between a sincos per dipole and the tables; one direction is two kernels"""
    import adda_gb300 as A
    s = full_box(shape, 2 * math.pi)
    x = random_vec(s.n, R, 3)
    d = some_dirs(max(dirs), 9)
    pick = sorted({0, 1, 4, 5, 6, 30, 32, 39, 339, 359} & set(range(max(dirs))))
    for n in dirs:
        e, P = fields_of(s, x, d[:n], 0)
        if n == dirs[0]:
            want = fields_direct(s, P, d[pick])
        q = [i for i, v in enumerate(pick) if v < n]
        err = field_errors(e[:, [pick[i] for i in q]], want[:, q])
        assert np.sqrt((err ** 2).mean()) < FIELD_TOL
    # launches of the call alone
    c = context(s, R=R)
    import torch
    d_x = torch.from_numpy(x.view(np.float64)).cuda()
    torch.cuda.synchronize()
    c.solve_device(d_x.data_ptr(), R, d_x.data_ptr(), prec="fp64", maxiter=0, init="x0")
    before = A.kernel_launches()
    c.scattered_fields(d[:1], R)
    assert A.kernel_launches() - before == 2
    c.close()


def test_fields_of_few_directions_in_a_group():
    """every particle of a group context sums its own dipoles"""
    import torch

    import adda_gb300 as A
    ss = [A.Setup(grid=g, shape="ellipsoid", pars=(0.8, 0.6), m=1.4 + 0.05j, dpl=12) for g in (12, 8)]
    c = A.Context.group(ss, rhs_per_particle=2)
    x = np.zeros((4, 3 * c.n), complex)
    for r in range(4):
        c.set_cc(r, np.ones((1, 3)))
        x[r] = c.group_pad(random_vec(ss[r // 2].n, 1, r)[0], r // 2).reshape(-1)
    c.init_dmatrix()
    d_x = torch.from_numpy(x.view(np.float64)).cuda()
    torch.cuda.synchronize()
    c.solve_device(d_x.data_ptr(), 4, d_x.data_ptr(), prec="fp64", maxiter=0, init="x0")
    d = some_dirs(2, 4)
    e = c.scattered_fields(d, 4)
    many = c.scattered_fields(np.concatenate([d, some_dirs(2000, 5)]), 4)[:, :2]
    assert field_errors(e, many.astype(CLD)).max() < 2 * FIELD_TOL
    c.close()


# ---------------------------------------------------------------------------------------------------------------------
def test_cross_sections_do_not_depend_on_the_solve_before():
    """the same polarisations give the same digits after an FP64 and after a mixed-precision solve"""
    import torch

    import adda_gb300 as A
    s = A.Setup(grid=24, m=1.4 + 0.02j, dpl=12)
    c = context(s, R=2)
    prop, pol, e = np.stack([s.prop] * 2), np.stack(s.incpol), np.stack(s.einc)
    for prec in ("mixed", "mixed_f32vec"):
        res = c.solve(e, prec=prec, eps=1e-3)
        got = [c.cross_sections(prop, pol), c.cross_sections_beam(e)]
        d_x = torch.from_numpy(res["x"].view(np.float64)).cuda()
        d_p = torch.empty_like(d_x)
        torch.cuda.synchronize()
        c.solve_device(d_x.data_ptr(), 2, d_x.data_ptr(), d_p.data_ptr(), prec="fp64", maxiter=0, init="x0")
        torch.cuda.synchronize()
        assert np.array_equal(d_p.cpu().numpy().view(np.complex128).reshape(2, -1), res["p"])
        assert np.array_equal(np.array([c.cross_sections(prop, pol), c.cross_sections_beam(e)]), np.array(got))
    c.close()


@pytest.mark.parametrize("surface", [False, True])
def test_one_copy_of_the_interaction_matrix(surface):
    """a context holds the FP64 matrix in one form: 16 + 8 bytes an entry, and the matvec's and vectors' buffers"""
    import torch

    import adda_gb300 as A
    s = full_box((3, 126, 126), 1.0)
    s.grid = (300, 252, 252) if not surface else (150, 252, 252)
    kw = dict(surface=dict(zsum_shift=1.25, msub=1.5 + 0.1j, relation="img")) if surface else {}
    A.Context((2, 2, 2), full_box((2, 2, 2), 1.0).pos, None, 0.4, 1.0, (4, 4, 4)).close()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    c = A.Context(s.box, s.pos, s.mat, s.gridspace, 1.0, s.grid, nrhs_max=1, **kw)
    c.init_dmatrix()
    torch.cuda.synchronize()
    used = free - torch.cuda.mem_get_info()[0]
    g, b = s.grid, s.box
    entries = 6 * g[0] * (g[1] // 2 + 1) * (g[2] // 2 + 1) + (6 * g[0] * (g[1] // 2 + 1) * g[2] if surface else 0)
    slab = 3 * g[2] * b[1]
    chunk = (4 if surface else 2) * max(48 << 20, 8 * slab * g[0])
    work = 16 * 3 * g[0] * b[1] * b[2] + chunk + 2 * 16 * 3 * s.n
    assert 24 * entries > 4 * (64 << 20) and used < 24 * entries * 1.02 + work + (64 << 20)
    c.close()


@pytest.mark.parametrize("surface", [False, True])
def test_forms_of_the_interaction_matrix(surface):
    """reading the matrix back, and tile shapes that take the FP64 transforms and back, before and after it is built, leave
    the matrix and the matvec as they are"""
    import adda_gb300 as A
    s = full_box((10, 7, 6), 1.0)
    kw = dict(surface=dict(zsum_shift=1.25, msub=1.5 + 0.1j, relation="img")) if surface else {}

    def make(shape=None):
        c = A.Context(s.box, s.pos, s.mat, s.gridspace, 1.0, s.grid, nrhs_max=2, **kw)
        if shape:
            c.set_fft_shape(shape, "fp64")
        c.init_dmatrix()
        for r in range(2):
            c.set_cc(r, s.cc[r].reshape(1, 3))
        return c

    x = random_vec(s.n, 2, 1)
    c = make()
    plain, narrow = list(c.fft_shape("fp64")), [1] + list(c.fft_shape("fp64"))[1:]
    y = c.matvec(x, "fp64")[0]
    d, r = c.dmatrix(), c.rmatrix() if surface else None
    assert np.array_equal(c.matvec(x, "fp64")[0], y) and np.array_equal(c.dmatrix(), d)
    c.set_fft_shape(narrow, "fp64")
    y64 = c.matvec(x, "fp64")[0]
    assert 0 < np.abs(y64 - y).max() < 1e-14 * np.abs(y).max()
    c.set_fft_shape(plain, "fp64")
    assert np.array_equal(c.matvec(x, "fp64")[0], y)
    c.init_dmatrix()
    assert np.array_equal(c.matvec(x, "fp64")[0], y) and np.array_equal(c.dmatrix(), d)
    n = make(narrow)
    assert np.array_equal(n.matvec(x, "fp64")[0], y64) and np.array_equal(n.dmatrix(), d)
    n.set_fft_shape(plain, "fp64")
    assert np.array_equal(n.matvec(x, "fp64")[0], y) and np.array_equal(n.dmatrix(), d)
    if surface:
        assert np.array_equal(c.rmatrix(), r) and np.array_equal(n.rmatrix(), r)
    n.set_fft_shape(narrow, "fp64")
    n.init_dmatrix()
    assert np.array_equal(n.matvec(x, "fp64")[0], y64)
    c.close()
    n.close()


@pytest.mark.parametrize("box", [(16, 16, 8), (32, 4, 30)])
def test_block_sums_round(box):
    """|y|^2 of y = x (polarisabilities of 1e-300) where each warp sums one value of 1 and others 2^-17 of it that end just
    below the sum's unit of 2^-56. Cut off, they would all be short by one: 31 * 2^-56 = 4.3e-16. Bound: the block's and the
    total's rounding to a double, 2 * 2^-53"""
    s = full_box(box, 1.0)
    s.cc = [np.full(3, 1e-300)] * 2
    c = context(s, R=1)
    b = next(v for v in range((1 << 26) + 1, 1 << 27, 2) if v * v < 1 << 53 and v * v % 4096 == 4089)
    x = np.zeros((1, s.n, 3), complex)
    x[0, :, 0] = b * 2.0 ** -26 * 2.0 ** -8
    x[0, ::32, 0] = 1
    y, ip = c.matvec(x.reshape(1, -1), "fp64")
    y = y.reshape(x.shape)
    assert np.array_equal(y[..., 0].real, x[..., 0].real) and max(abs(y.imag).max(), abs(y[..., 1:]).max()) < 1e-200
    want = math.fsum((x.real ** 2).ravel())
    assert abs(ip[0] - want) <= 2.3e-16 * want
    c.close()


# ---------------------------------------------------------------------------------------------------------------------
# The fixed-point transforms at the ends of their range

@pytest.mark.parametrize("n", [64, 256, 384, 400, 500, 512])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_coherent_input_on_a_long_axis(axis, n):
    """constants and plane waves put a line's spectrum into one element, the largest growth of the forward transform (n / 2
    terms of one sign: radices 16 x 16, 16 x 24, 20 x 25, 16 x 32, shifts of 2 and 3 bits); a single dipole has a flat
    spectrum, the largest of the inverse ones (n terms). An overflow would be an error of the order of the result"""
    from helpers import oracle_for, rel
    box = [3, 2, 3]
    box[axis] = n // 2
    s = cube_setup(box, [2 * b for b in box])
    s.cc = [s.cc[0]] * 2
    o, c = oracle_for(s), context(s, R=6)
    o.set_cc(s.cc[0].reshape(1, 3))
    pol = np.array([1.0, 1.0j, -1.0])
    along = s.pos[:, axis].astype(float)
    x = [np.exp(2j * np.pi * f / n * along)[:, None] * pol for f in (0, n // 4, n // 2 - 1)]
    for at in (0, n // 4, n // 2 - 1):
        d = np.zeros((s.n, 3), complex)
        d[np.flatnonzero(s.pos[:, axis] == at)[0]] = pol
        x.append(d)
    x = np.stack(x).reshape(6, -1)
    for her in (False, True):
        y = c.matvec(x, "fp64", her)[0]
        for r in range(6):
            assert rel(y[r], o.matvec(x[r], her)[0]) < 6e-15, (r, her)
    o.close()
    c.close()


@pytest.mark.parametrize("box", [(32, 32, 32), (64, 45, 40), (100, 20, 16), (12, 125, 10)])
@pytest.mark.parametrize("scale", [(1, 1, 1), (1, 1e-4, 1e-8), (1e-8, 1, 1e-4)])
def test_fp64_matvec_to_rounding(box, scale):
    """errors of twelve dipoles against a direct sum in extended precision, relative to the result's rms"""
    s = full_box(box, 1.0)
    c = context(s, R=1)
    x = random_vec(s.n, 1, 17).reshape(s.n, 3) * np.array(scale)
    y = c.matvec(x.reshape(1, -1), "fp64")[0].reshape(s.n, 3)
    pick = np.random.default_rng(3).choice(s.n, 12, replace=False)
    err = np.abs(y[pick] - matvec_direct(s, s.cc[0], x, pick)).astype(float)
    assert np.sqrt((err ** 2).sum(1).mean() / (np.abs(y) ** 2).sum(1).mean()) < TOL
    c.close()


@pytest.mark.parametrize("n", [9, 15, 21, 25, 27, 35, 49, 63, 77, 105, 121, 125, 143, 169, 195, 225, 243, 315, 375])
def test_odd_x_grids(n):
    """an x axis of 2 boxX - 1 points: the two-pass transforms' zero half is a point short of half the line"""
    from helpers import oracle_for, rel
    s = cube_setup(((n + 1) // 2, 3, 2), (n, 6, 4))
    s.cc = [s.cc[0]] * 2
    o, c = oracle_for(s), context(s, R=2)
    o.set_cc(s.cc[0].reshape(1, 3))
    x = random_vec(s.n, 2, n)
    for prec, tol in (("fp64", 6e-15), ("fp32", 5e-6)):
        y = c.matvec(x, prec)[0]
        for r in range(2):
            assert rel(y[r], o.matvec(x[r])[0]) < tol
    o.close()
    c.close()


@pytest.mark.parametrize("method", ["bicg", "cgnr", "csym", "qmr2", "bcgs2"])
@pytest.mark.parametrize("grid", [6, 10, 16])
def test_other_methods_of_few_and_many_blocks(method, grid):
    """vector kernels of one block, a few and dozens per right-hand side, scalar steps in the last block or as kernels: several
    right-hand sides of different scale converge independently to the oracle's solution"""
    from oracle import oracle as O

    from helpers import oracle_for, rel, setup_for
    s = setup_for(dict(grid=grid, m=1.3 + 0.1j, dpl=10))
    o, c = oracle_for(s), context(s, R=3)
    scale = [1.0, 1e-30, 1e30]
    for r in range(3):
        c.set_cc(r, s.cc[0].reshape(1, 3))
    o.set_cc(s.cc[0].reshape(1, 3))
    want = o.solve(s.einc[0], method=O.QMR_CS, eps=1e-11)["p"]
    res = c.solve(np.stack([s.einc[0] * k for k in scale]), method=method, prec="fp64", eps=1e-11)
    for r in range(3):
        assert res["stats"][r]["status"] == "ok", (r, res["stats"][r])
        # the relative error is at most the condition number (below 10 for m = 1.3) times the residual
        assert rel(res["p"][r] / scale[r], want) < 1e-9
    o.close()
    c.close()
