"""Position derivatives of cells with as many edges as eight lanes take in
one, two and eight turns, and past the capacity.

One Dirac inside a ring of m others has a cell of m edges.  The columns of its
own and of two neighbours' unknowns are compared with central differences of
the diagram's centroids and masses, step H = 1e-6: a vertex of the ring's cell
moves by at most H / (2 sin(pi / 64)) ~ 1e-5 against edges of at least 0.01, so
the differences' own error is (1e-3)^2 relative at the worst, and 1e-16 / H =
1e-10 by rounding; RTOL = 1e-5 of the largest entry of a column covers both."""
import numpy as np
import pytest

from sdot_b200.power_diagram import PowerDiagram

pytestmark = pytest.mark.gpu

H = 1e-6
RTOL = 1e-5


def ring(m):
    rng = np.random.default_rng(400 + m)
    a = 2 * np.pi * (np.arange(m) + 0.1 * rng.uniform(-1, 1, m)) / m
    r = 0.3 * (1 + 1e-4 * rng.uniform(-1, 1, m))
    p = 0.5 + np.stack([r * np.cos(a), r * np.sin(a)], 1)
    return np.concatenate([p, [[0.5, 0.5]]])


def diagram(p, w):
    g = PowerDiagram(p, w)
    g.add_box_shape([0, 0], [1, 1])
    return g


def values(p, w):
    c, m = diagram(p, w).centroids(with_masses=True)
    return np.concatenate([c, m[:, None]], 1).ravel()


@pytest.mark.parametrize("m", [7, 8, 9, 16, 17, 63, 64])
def test_derpos_ring(gpu_lib, m):
    p, w = ring(m), np.zeros(m + 1)
    off, col, val, v = diagram(p, w).der_centroids_and_integrals_wrt_weight_and_positions()
    assert off[3 * m + 1] - off[3 * m] == 3 * (m + 1), "the inner cell's edges"
    assert np.allclose(v, values(p, w), rtol=0, atol=1e-13)
    rows = np.repeat(np.arange(3 * m + 3), np.diff(off))
    for r in range(3 * m + 3):
        assert np.all(np.diff(col[off[r]:off[r + 1]]) > 0)
    for i in (m, 0, m // 2):
        for e in range(3):
            d = []
            for h in (H, -H):
                q, u = p.copy(), w.copy()
                if e < 2:
                    q[i, e] += h
                else:
                    u[i] += h
                d.append(values(q, u))
            fd = (d[0] - d[1]) / (2 * H)
            got = np.zeros(3 * m + 3)
            sel = col == 3 * i + e
            got[rows[sel]] = val[sel]
            for k in range(3):
                scale = np.abs(fd[k::3]).max()
                assert np.abs(got[k::3] - fd[k::3]).max() <= RTOL * scale, (i, e, k)


def test_derpos_past_capacity(gpu_lib):
    with pytest.raises(Exception):
        diagram(ring(65), np.zeros(66)).der_centroids_and_integrals_wrt_weight_and_positions()
