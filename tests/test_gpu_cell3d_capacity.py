"""3D cells at the edges of the passes' capacities (64 vertices and faces, then
192 vertices and 128 faces, then 256 faces), against the qhull oracle
(oracle/poly3d.py).  One Dirac at the centre of k others on a sphere has a cell
of k faces and 2 k - 4 vertices; with the six box faces cut away on the way it
passes through k + 6 faces at most.  Tolerances as the other tests against this
oracle: 1e-11 relative to max(|value|, a tenth of the mean)."""
import numpy as np
import pytest

from sdot_b200._lib import SDOT_CAPACITY, SdotError
from sdot_b200.power_diagram import PowerDiagram

pytestmark = pytest.mark.gpu


def sphere(k, seed=0):
    """k nearly evenly spread points at distances 0.4 (1 +- 1e-3) of the box's
    centre (a golden-angle spiral, jittered), and the centre.  (At one distance
    every bisector of two of them would pass through the centre: cuts decided
    by rounding.)"""
    rng = np.random.default_rng(7000 + seed + k)
    z = 1 - (2 * np.arange(k) + 1) / k
    a = np.pi * (3 - np.sqrt(5)) * np.arange(k)
    r = np.sqrt(1 - z * z)
    d = np.stack([r * np.cos(a), r * np.sin(a), z], 1) + rng.normal(scale=0.05 / np.sqrt(k), size=(k, 3))
    d *= (0.4 * rng.uniform(0.999, 1.001, k) / np.linalg.norm(d, axis=1))[:, None]
    return np.concatenate([[[0.5, 0.5, 0.5]], 0.5 + d])


def diagram(p):
    g = PowerDiagram(p, np.zeros(len(p)))
    g.add_box_shape(np.zeros(3), np.ones(3))
    return g


@pytest.mark.parametrize("k", [4, 13, 17, 33, 34, 35, 63, 66, 97, 99, 127, 130, 249])
def test_faces_of_one_cell(gpu_lib, k):
    from oracle import poly3d

    p = sphere(k)
    g = diagram(p)
    m_o, c_o, H_o = poly3d.integrate(p, np.zeros(k + 1))
    m = g.integrals()
    np.testing.assert_allclose(m, m_o, rtol=1e-11, atol=1e-12 * m_o.mean())
    np.testing.assert_allclose(g.centroids(), c_o, rtol=1e-11, atol=1e-12)
    assert abs(m.sum() - 1.0) < 1e-12
    off, col, val, _ = g.der_integrals_wrt_weights()
    H = {(i, int(col[q])): val[q] for i in range(k + 1) for q in range(off[i], off[i + 1])}
    scale = max(abs(v) for v in H_o.values())
    assert max(abs(H.get(q, 0.0) - H_o.get(q, 0.0)) for q in set(H) | set(H_o)) < 1e-11 * scale
    # a second evaluation goes by the pass each cell needed
    g.set_weights(np.zeros(k + 1))
    assert np.array_equal(g.integrals(), m)


def test_more_faces_than_the_last_pass(gpu_lib):
    with pytest.raises(SdotError) as e:
        diagram(sphere(300)).integrals()
    assert e.value.status == SDOT_CAPACITY
