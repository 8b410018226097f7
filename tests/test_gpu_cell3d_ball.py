"""3D cells at scales where the squares that the ball tests compare stay in
range, and where they do not (2^-250, 2^250: the vertices decide alone).

Scaling by a power of two is exact, so masses and neighbours must not depend on
the scale but for the order of the cuts (the keys of the boxes are floats, which
run out of range): RTOL = 1e-12 of the mean mass, as elsewhere.  The cells tile
the box (their masses sum to it within n times that) and a neighbour's
neighbours hold the cell: a cut that one of two cells misses breaks both."""
import numpy as np
import pytest

from sdot_b200.power_diagram import PowerDiagram

pytestmark = pytest.mark.gpu

RTOL = 1e-12


def inputs(kind, n):
    rng = np.random.default_rng(500)
    p = rng.random((n, 3))
    w = np.zeros(n)
    if kind == "weights":
        w = rng.uniform(-1, 1, n) * n ** (-2 / 3) * 0.3
    elif kind == "one large":
        w[n // 2] = 0.04
    elif kind == "offset":
        w = 1e3 + rng.uniform(-1, 1, n) * 1e-3
    return p, w


def run(p, w, k):
    g = PowerDiagram(p * 2.0 ** k, w * 2.0 ** (2 * k))
    g.add_box_shape([0, 0, 0], [2.0 ** k] * 3)
    off, ids = g.neighbors()
    return g.integrals() / 2.0 ** (3 * k), off, ids


@pytest.mark.parametrize("kind", ["zero", "weights", "one large", "offset"])
@pytest.mark.parametrize("n", [2, 60, 700])
def test_cells3d_scales(gpu_lib, kind, n):
    p, w = inputs(kind, n)
    m0, o0, i0 = run(p, w, 0)
    assert abs(m0.sum() - 1) <= RTOL * n
    pairs = {(i, j) for i in range(n) for j in i0[o0[i]:o0[i + 1]] if j >= 0}
    assert all((j, i) in pairs for i, j in pairs)
    for k in (-250, -60, 60, 250):
        m, o, i = run(p, w, k)
        assert np.abs(m - m0).max() <= RTOL / n
        assert np.array_equal(o, o0)
        for c in range(n):
            assert sorted(i[o[c]:o[c + 1]]) == sorted(i0[o0[c]:o0[c + 1]])
