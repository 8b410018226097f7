"""2D cells at the edges of the fast tier's storage (polygons of 13 vertices,
kept as an order over slots) and of its warps and blocks, against the C
restatement (oracle/port.py), with the bounds of the 2D parity tests: 1e-12 of
max(|value|, mean), 1e-11 for the Hessian of the near-circular cell, whose short
edges are differences of nearby vertices."""
import numpy as np
import pytest

from oracle import port
from sdot_b200.power_diagram import PowerDiagram
from tests.test_gpu_parity_2d import check_all

pytestmark = pytest.mark.gpu


def pair(p, w, image=None, **kw):
    out = []
    for cls in (PowerDiagram, port.PortPowerDiagram):
        d = cls(p, w, **kw)
        if image is None:
            d.add_box_shape([0.0, 0.0], [1.0, 1.0])
        else:
            d.set_image_density(image)
        out.append(d)
    return out


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("k", list(range(3, 18)) + [40])
def test_edges_of_one_cell(gpu_lib, k, precision):
    # one cell of k edges: cuts that remove one, two and more vertices, over
    # vertex 0 too (the Diracs' order is random), up to and past 13 vertices
    rng = np.random.default_rng(8100 + k)
    a = rng.permutation(k) * 2 * np.pi / k + rng.uniform(-0.3, 0.3, k) / k
    d = 0.4 * rng.uniform(0.999, 1.001, k)
    p = np.concatenate([[[0.5, 0.5]], 0.5 + d[:, None] * np.stack([np.cos(a), np.sin(a)], 1)])
    g, r = pair(p, np.zeros(k + 1))
    if precision == "mixed":
        g = PowerDiagram(p, np.zeros(k + 1), precision="mixed")
        g.add_box_shape([0.0, 0.0], [1.0, 1.0])
    check_all(g, r, k + 1, rtol_hess=1e-11)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 127, 129, 1025, 6000, 6001, 16384, 16386, 16417])
def test_walks_of_one_warp(gpu_lib, n):
    # lanes whose walks end far apart: weights that empty some cells and make
    # others reach over many, and a last warp of a few lanes; a warp per cell up
    # to 6,000 Diracs, warps of 12 cells up to 16,384
    rng = np.random.default_rng(8200 + n)
    g, r = pair(rng.random((n, 2)), rng.uniform(-1.0, 1.0, n) / n)
    check_all(g, r, n, rtol_hess=1e-11)


@pytest.mark.parametrize("k", [13, 47, 48, 49, 63, 64, 65, 200])
def test_large_cells_among_many(gpu_lib, k):
    # cells past the fast tier in a diagram that starts there, around the
    # capacity of the warps' shared memory: a ring of k Diracs about one in the
    # middle of 7,000 others, which are kept out of the ring
    rng = np.random.default_rng(8400 + k)
    q = rng.random((12000, 2))
    q = q[np.hypot(q[:, 0] - 0.5, q[:, 1] - 0.5) > 0.35][:7000]
    a = np.arange(k) * 2 * np.pi / k + rng.uniform(-0.2, 0.2, k) / k
    d = 0.25 * rng.uniform(0.9999, 1.0001, k)
    p = np.concatenate([q, 0.5 + d[:, None] * np.stack([np.cos(a), np.sin(a)], 1), [[0.5, 0.5]]])
    g, r = pair(p, np.zeros(len(p)))
    check_all(g, r, len(p), rtol_hess=1e-11)


@pytest.mark.parametrize("n,res", [(1, (1, 1)), (3, (40, 7)), (40, (3, 5)), (300, (64, 64)), (2000, (5, 90))])
@pytest.mark.parametrize("disc", [None, 0.2, 4.0])
def test_pieces_of_pixels(gpu_lib, n, res, disc):
    # pixels much larger and much smaller than the cells, cells cut by none to
    # all four lines of a pixel, discs inside their cells and around them (the
    # arcs' functions differ by a few ulp between device and host: 1e-11)
    rng = np.random.default_rng(8300 + n)
    w = rng.uniform(-0.1, 0.1, n) / n if disc is None else disc / n * rng.uniform(0.5, 2.0, n)
    g, r = pair(rng.random((n, 2)), w, image=rng.uniform(0.5, 1.5, res),
                radial_func="unit" if disc is None else "in_ball_w05")
    check_all(g, r, n, rtol=1e-12 if disc is None else 1e-11, rtol_hess=1e-11)
