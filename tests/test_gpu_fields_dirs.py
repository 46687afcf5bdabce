"""Scattered fields against a direct sum in numpy over the number of directions (one warp of 32 and its edges, the splits
of the dipoles between warps, several launches of the direction tables' budget), the RHS count and particles whose lines
are longer than one run of the fixed-point sums (128 dipoles).

Tolerance: the phase's argument, up to kd * |n.pos| < 400 rad here, is rounded to 2^-53 of it on both sides, by up to three
roundings: 3 * 400 * 2^-53 = 1.4e-13 a term at most, random in sign over the dipoles, on sums not smaller than the
terms' rms: 2e-13 of the largest field."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solved(shape, grid, pars, R, seed):
    """a context whose polarisations are cc_sqrt * x for a given x (no iterations)"""
    import torch

    import adda_gb300 as A
    s = A.Setup(grid=grid, shape=shape, pars=pars, m=1.3 + 0.05j, dpl=10)
    c = A.Context(s.box, s.pos, s.mat, s.gridspace, s.wavenum, s.grid, nrhs_max=R)
    c.init_dmatrix()
    for r in range(R):
        c.set_cc(r, s.cc[r % 2].reshape(1, 3))
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((R, 3 * s.n)) + 1j * rng.standard_normal((R, 3 * s.n))
    d_x = torch.from_numpy(x.view(np.float64)).cuda()
    torch.cuda.synchronize()
    c.solve_device(d_x.data_ptr(), R, d_x.data_ptr(), prec="fp64", maxiter=0, init="x0")
    P = np.stack([x[r].reshape(-1, 3) * np.sqrt(s.cc[r % 2]) for r in range(R)])
    return s, c, P


def direct(s, P, dirs):
    pos = s.pos.astype(np.float64) - (np.array(s.box) - 1) / 2
    w = np.exp(-1j * s.kd * (dirs @ pos.T))
    f = np.einsum("dn,rnc->rdc", w, P)
    return -1j * s.wavenum ** 3 * (f - dirs * np.einsum("rdc,dc->rd", f, dirs)[..., None])


@pytest.mark.parametrize("ndir", [1, 31, 32, 33, 64, 100, 129, 500])
@pytest.mark.parametrize("shape,grid,pars,R", [("sphere", 12, None, 1), ("box", 300, (0.01, 0.014), 2),
                                               ("ellipsoid", 20, (0.7, 0.55), 3)])
def test_fields_match_direct_sum(shape, grid, pars, R, ndir):
    s, c, P = solved(shape, grid, pars, R, ndir)
    d = np.random.default_rng(ndir).standard_normal((ndir, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    want = direct(s, P, d)
    assert np.abs(c.scattered_fields(d, R) - want).max() < 2e-13 * np.abs(want).max()
    c.close()


def test_many_directions_need_several_tables():
    """a box 300 long has over 300 table rows: about 13 500 directions per launch"""
    s, c, P = solved("box", 300, (0.01, 0.014), 1, 5)
    d = np.random.default_rng(0).standard_normal((20000, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    got = c.scattered_fields(d, 1)
    pick = [0, 1, 13503, 13504, 13535, 13536, 19999]
    want = direct(s, P, d[pick])
    assert np.abs(got[:, pick] - want).max() < 2e-13 * np.abs(want).max()
    c.close()


def test_non_finite_polarisation():
    s, c, P = solved("sphere", 8, None, 2, 1)
    import torch
    x = np.zeros((2, 3 * s.n), complex)
    x[0, 3], x[1, 5] = np.nan, 1.0
    d_x = torch.from_numpy(x.view(np.float64)).cuda()
    torch.cuda.synchronize()
    c.solve_device(d_x.data_ptr(), 2, d_x.data_ptr(), prec="fp64", maxiter=0, init="x0")
    e = c.scattered_fields(np.eye(3), 2)
    assert np.isnan(e[0]).all() and np.isfinite(e[1]).all() and e[1].any()
    c.close()
