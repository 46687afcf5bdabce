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


def matvec_direct(s, cc, x):
    """x - S G S x by a direct sum over the dipoles in extended precision, [n, 3]"""
    S = np.sqrt(cc.reshape(-1)[:3].astype(CLD))
    v = x * S
    pos, out = s.pos.astype(LD), np.empty((s.n, 3), CLD)
    kd = LD(s.wavenum) * LD(s.gridspace)
    for i in range(s.n):
        d = pos[i] - pos
        d[i] = 1
        r = np.sqrt((d * d).sum(1))
        q, kr = d / r[:, None], kd * r
        e = np.exp(1j * kr.astype(CLD)) / (LD(s.gridspace) * r) ** 3
        e[i] = 0
        a, b = e * (kr * kr - 1 + 1j * kr), e * (3 - kr * kr - 3j * kr) * (q * v).sum(1)
        out[i] = x[i] - S * (a[:, None] * v + b[:, None] * q).sum(0)
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
