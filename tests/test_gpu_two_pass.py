"""The matvec on two-pass transforms (axis lengths n = r1*r2 with radices up to 32): the FP64 matvec, in 64-bit fixed
point, and the FP32 matvec of lengths without compile-time kernels.

FP64 tolerance: a transform adds noise of about 2^-54 of its block's largest value, six transforms and the D product
follow one another, and the largest value of these random data is below 16 times their rms: 7 * 16 * 2^-54 = 6e-15.
FP32: the 5e-6 of the other parity tests."""
import numpy as np
import pytest

from helpers import oracle_for, rel, setup_for
from test_gpu_parity import context, cube_setup, random_vec

pytestmark = pytest.mark.gpu
TOL64, TOL32 = 6e-15, 5e-6

# lengths whose plans hold every radix in the first or the second pass
LENGTHS = [2, 4, 6, 10, 14, 18, 22, 26, 32, 36, 44, 52, 70, 78, 80, 90, 96, 98, 110, 130, 132, 154, 156, 168, 180, 182,
           196, 208, 210, 224, 240, 256]
# radices above 16 (FP32: 18 to 32; fixed point: 18, 20, 24, 25, 32, the other lengths fall back to FP64 instructions)
LENGTHS += [162, 198, 200, 216, 220, 234, 250, 252, 264, 288, 294, 300, 308, 324, 336, 350, 352, 360, 364, 378, 390, 396,
            400, 416, 432, 448, 450, 480, 486, 500, 512]


def check(s, x, her=False, precs=("fp64", "fp32")):
    o, c = oracle_for(s), context(s, R=x.shape[0])
    for prec in precs:
        y, ip = c.matvec(x, prec, her)
        for r in range(x.shape[0]):
            o.set_cc(s.cc[r % 2].reshape(1, 3))
            yr, ipr = o.matvec(x[r], her)
            assert rel(y[r], yr) < (TOL64 if prec == "fp64" else TOL32), (prec, r)
            assert abs(ip[r] / ipr - 1) < (1e-12 if prec == "fp64" else 1e-5)
    o.close()
    c.close()


@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_axis_length(axis, n):
    """a thin box with the length along one axis (full to half of it, and with a ragged particle edge)"""
    box, grid = [3, 2, 3], [6, 4, 6]
    box[axis], grid[axis] = n // 2, n
    s = cube_setup(box, grid)
    check(s, random_vec(s.n, 2, n + axis), her=bool(n % 4))


def test_scales_zeros_and_tiny_values():
    """right-hand sides of very different magnitude, zeros and subnormal numbers keep their own exponents"""
    s = setup_for(dict(grid=16, m=1.5, dpl=10))
    x = random_vec(s.n, 1, 3)[0]
    scales = [1.0, 1e-200, 1e200, 2.0 ** -1060]
    c = context(s, R=6)
    y, _ = c.matvec(np.stack([x * k for k in scales] + [np.zeros_like(x), x]), "fp64")
    assert rel(y[1] * 1e200, y[0]) < TOL64 and rel(y[2] * 1e-200, y[0]) < TOL64
    # spacing 2^-1074: the input itself has about 14 bits
    assert rel(y[3] * 2.0 ** 1000 * 2.0 ** 60, y[0]) < 1e-3
    assert not y[4].any() and np.array_equal(y[5], y[0])
    c.close()


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_non_finite_input_stays_with_its_rhs(bad):
    s = setup_for(dict(grid=16, m=1.5, dpl=10))
    x = random_vec(s.n, 2, 4)
    c = context(s, R=2)
    good, _ = c.matvec(x, "fp64")
    x[1, 17] = bad
    y, _ = c.matvec(x, "fp64")
    assert np.array_equal(y[0], good[0]) and np.isnan(y[1]).all()
    again, _ = c.matvec(np.stack([x[0], x[0]]), "fp64")
    assert rel(again[0], good[0]) == 0 and np.isfinite(again[1]).all()
    c.close()


def test_concentrated_spectrum():
    """a plane wave along an axis of a full cube puts the whole spectrum into a few elements: the transforms reach the
    largest growth their range allows"""
    s = cube_setup((32, 32, 32), (64, 64, 64))
    k = 2 * np.pi / 64 * np.array([[0, 0, 0], [8, 0, 0], [16, 16, 0], [31, 31, 31]])
    pol = np.array([1.0, 1.0j, -1.0])
    x = np.stack([(np.exp(1j * s.pos @ kk)[:, None] * pol).reshape(-1) for kk in k])
    check(s, x, precs=("fp64",))


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_block_sums_of_extreme_values(prec):
    """|y|^2 (block sums in fixed point relative to a warp's largest value) of vectors of very different magnitude, of a
    vector with one large element among tiny ones, of zeros, and of vectors with NaN and infinity"""
    s = setup_for(dict(grid=16, m=1.5, dpl=10))
    x = random_vec(s.n, 1, 8)[0]
    big = 1e15 if prec == "fp32" else 1e100
    spike = x * (1e-12 / big)
    spike[5] = big
    bad = [x.copy(), x.copy()]
    bad[0][3], bad[1][4] = np.nan, np.inf
    c = context(s, R=7)
    y, ip = c.matvec(np.stack([x, x * big, x / big, spike, np.zeros_like(x)] + bad), prec)
    for r in range(4):
        # the FP32 sums are of the rounded results in double: both to rounding
        assert abs(ip[r] / np.sum(np.abs(y[r]) ** 2) - 1) < 1e-12
    assert ip[4] == 0 and not np.isfinite(ip[5:]).any()
    c.close()


@pytest.mark.parametrize("method", ["qmr", "bicgstab"])
@pytest.mark.parametrize("grid", [2, 4, 6, 10])
def test_scalar_steps_in_the_last_block(method, grid):
    """solves whose vector kernels have one block, and a few, per right-hand side; several right-hand sides of different
    scale converge independently to the oracle's solution"""
    from oracle import oracle as O
    s = setup_for(dict(grid=grid, m=1.3 + 0.1j, dpl=10))
    o, c = oracle_for(s), context(s, R=3)
    scale = [1.0, 1e-30, 1e30]
    e = np.stack([s.einc[0] * k for k in scale])
    for r in range(3):
        c.set_cc(r, s.cc[0].reshape(1, 3))
    o.set_cc(s.cc[0].reshape(1, 3))
    want = o.solve(s.einc[0], method={"qmr": O.QMR_CS, "bicgstab": O.BICGSTAB}[method], eps=1e-11)["p"]
    res = c.solve(e, method=method, prec="fp64", eps=1e-11)
    for r in range(3):
        assert res["stats"][r]["status"] == "ok"
        assert rel(res["p"][r] / scale[r], want) < 1e-9
    o.close()
    c.close()


@pytest.mark.parametrize("box", [(6, 5, 4), (11, 9, 13), (32, 32, 32), (25, 10, 45), (7, 100, 6), (6, 5, 110)])
def test_particle_near_a_substrate(box):
    """the reflected transform and product: small and large radices, odd boxes, a power-of-two grid"""
    import adda_gb300 as A
    s = cube_setup(box, tuple(A.fft_fit(2 * v, 2) for v in box))
    s.surface = dict(zsum_shift=1.25, msub=1.5 + 0.1j, relation="img")
    o = oracle_for(s)
    c = A.Context(s.box, s.pos, s.mat, s.gridspace, s.wavenum, s.grid, nrhs_max=2, surface=s.surface)
    c.init_dmatrix()
    x = random_vec(s.n, 2, sum(box))
    for r in range(2):
        c.set_cc(r, s.cc[r].reshape(1, 3))
    for her in (False, True):
        y, yf = c.matvec(x, "fp64", her)[0], c.matvec(x, "fp32", her)[0]
        for r in range(2):
            o.set_cc(s.cc[r].reshape(1, 3))
            yr = o.matvec(x[r], her)[0]
            assert rel(y[r], yr) < TOL64 and rel(yf[r], yr) < TOL32
    o.close()
    c.close()
