"""Hessian rows at the lengths where their sorting changes hands (8 lanes with
up to 32 entries, a warp with up to 256, one lane), with and without equal
columns to merge.

One Dirac inside a ring of m others has a row of m + 1 entries.  An entry is
half the edge's length over the distance, symmetric, and every row sums to zero:
each holds to a few hundred roundings, RTOL = 1e-11 of the largest entry.  The
same box given as two or three pieces meets every column once per piece: the
merged rows are those of the box, to the roundings of the pieces' edges."""
import numpy as np
import pytest

from sdot_b200.power_diagram import PowerDiagram

pytestmark = pytest.mark.gpu

RTOL = 1e-11


def ring(m):
    rng = np.random.default_rng(600 + m)
    a = 2 * np.pi * (np.arange(m) + 0.1 * rng.uniform(-1, 1, m)) / m
    r = 0.3 * (1 + 0.2 / m ** 2 * rng.uniform(-1, 1, m))
    p = 0.5 + np.stack([r * np.cos(a), r * np.sin(a)], 1)
    return rng.permutation(np.concatenate([p, [[0.5, 0.5]]]))


def rows(p, pieces):
    g = PowerDiagram(p, np.zeros(len(p)))
    x = np.linspace(0, 1, pieces + 1)
    for k in range(pieces):
        g.add_box_shape([x[k], 0], [x[k + 1], 1])
    off, col, val, _ = g.der_integrals_wrt_weights()
    for i in range(len(p)):
        assert np.all(np.diff(col[off[i]:off[i + 1]]) > 0), "columns ascend"
    return off, col, val


@pytest.mark.parametrize("m", [6, 7, 8, 15, 16, 31, 32, 33, 100, 255, 256, 300])
def test_rows_of_a_ring(gpu_lib, m):
    p = ring(m)
    off, col, val = rows(p, 1)
    hub = int(np.argmin(np.abs(p - 0.5).sum(1)))
    assert off[hub + 1] - off[hub] == m + 1
    scale = np.abs(val).max()
    r = np.repeat(np.arange(m + 1), np.diff(off))
    sums = np.zeros(m + 1)
    np.add.at(sums, r, val)
    assert np.abs(sums).max() <= RTOL * scale
    H = {(i, j): v for i, j, v in zip(r, col, val)}
    assert all(abs(v - H[j, i]) <= RTOL * scale for (i, j), v in H.items())
    for pieces in (2, 3):
        o, c, v = rows(p, pieces)
        assert np.array_equal(o, off) and np.array_equal(c, col)
        assert np.abs(v - val).max() <= RTOL * scale
