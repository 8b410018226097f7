"""Regular lattices of Diracs over images and rasters whose lines meet the
cells' sides: squares with corners split by rounding, sides on the pixels' lines.

A cell is a square of side h, and its integrals have closed forms.  Rounding: a
triangle of a piece is a sum of three products of up to X h, X the domain's
extent (5 u X h, u = 2^-53), which is 5 u m of a cell's area h^2 for m cells a
side; with at most 6 triangles a piece and 16 pieces a cell (9 pixels and what
lies an ulp beyond them) 480 u m, 1e-11 for the 192 cells of the largest."""
import numpy as np
import pytest

from sdot_b200.power_diagram import PowerDiagram

pytestmark = pytest.mark.gpu

TOL = 1e-11
BOXES = [(0.1, 0.8), (-0.3, 3.0), (0.0, 1.0), (-7.0, -6.1)]
# cells a side, pixels a side
SIZES = [(m, int(m * f)) for m in (50, 64, 100, 128) for f in (0.5, 1, 2, 3)] + [(96, 192), (150, 150), (192, 192)]


def lattice(m, lo, hi):
    """Positions (index i + m j for column i, row j, shuffled), the order, and h."""
    h = (hi - lo) / m
    g = lo + (np.arange(m) + 0.5) * h
    p = np.stack(np.meshgrid(g, g, indexing="xy"), -1).reshape(-1, 2)
    order = np.random.default_rng(m).permutation(m * m)
    return p[order], order, h


def cell_sums(a, m):
    """Sums of the (ny, nx) pixel values over each cell's pixels, (m, m); a
    pixel of more than one cell gives each its share."""
    r = a.shape[0]
    if r < m:
        f = m // r
        return np.repeat(np.repeat(a, f, 0), f, 1) / f ** 2
    f = r // m
    return a.reshape(m, f, m, f).sum((1, 3))


@pytest.mark.parametrize("m,res", SIZES)
@pytest.mark.parametrize("lo,hi", BOXES)
def test_constant_pixels(gpu_lib, m, res, lo, hi):
    p, order, h = lattice(m, lo, hi)
    img = np.random.default_rng(res).uniform(0.5, 1.5, (res, res))
    d = PowerDiagram(p, np.zeros(m * m))
    d.set_image_density(img, [lo, lo], [hi, hi])
    want = (cell_sums(img, m) * ((hi - lo) / res) ** 2).ravel()[order]
    assert np.abs(d.integrals() - want).max() <= TOL * h * h * 1.5
    c, mc = d.centroids(with_masses=True)
    assert np.abs(mc - want).max() <= TOL * h * h * 1.5
    x = lo + (np.arange(res) + 0.5) * (hi - lo) / res
    mid = cell_sums(img * x[None, :], m) / cell_sums(img, m) if res >= m else None
    if mid is not None:  # moments of size X m: X / h = m times the mass's error in units of h
        assert np.abs(c[:, 0] - mid.ravel()[order]).max() <= 3 * TOL * max(abs(lo), abs(hi))


@pytest.mark.parametrize("m,res", SIZES)
@pytest.mark.parametrize("lo,hi", BOXES[:2])
def test_quadratic_pixels(gpu_lib, m, res, lo, hi):
    p, order, h = lattice(m, lo, hi)
    q = np.random.default_rng(res).uniform(-0.02, 0.02, (6, res, res))
    q[0] += 1.0
    d = PowerDiagram(p, np.zeros(m * m))
    d.set_image_density(q, [lo, lo], [hi, hi], nb_coeffs=6)
    # integrals of 1, x, y, x^2, xy, y^2 over the rectangles cell x pixel
    k = max(m, res)
    e = lo + np.arange(k + 1) * ((hi - lo) / k)
    i0, i1, i2 = [np.diff(e ** (j + 1)) / (j + 1) for j in range(3)]
    r = np.repeat(np.repeat(q, k // res, 1), k // res, 2)
    one = [np.outer(i0, i0), np.outer(i0, i1), np.outer(i1, i0), np.outer(i0, i2), np.outer(i1, i1), np.outer(i2, i0)]
    dens = sum(r[j] * one[j] for j in range(6))
    f = k // m
    want = dens.reshape(m, f, m, f).sum((1, 3)).ravel()[order]
    assert np.abs(d.integrals() - want).max() <= TOL * h * h * 2


@pytest.mark.parametrize("m,res", SIZES)
@pytest.mark.parametrize("lo,hi", BOXES)
def test_rasters(gpu_lib, m, res, lo, hi):
    p, order, h = lattice(m, lo, hi)
    d = PowerDiagram(p, np.zeros(m * m))
    d.add_box_shape([lo, lo], [hi, hi])
    ps = (hi - lo) / res
    got = d.image_integrals([lo, lo], [hi, hi], (res, res))
    g = lo + (np.arange(m) + 0.5) * h
    k = max(m, res)
    f = k // res
    x = np.repeat(g, k // m).reshape(res, f).mean(1)  # mean position of a pixel's Diracs
    area = ps * ps
    assert np.abs(got[..., 2] - area).max() <= TOL * max(h * h, area)
    big = max(abs(lo), abs(hi))
    assert np.abs(got[..., 0] - area * x[None, :]).max() <= TOL * max(h * h, area) * big
    assert np.abs(got[..., 1] - area * x[:, None]).max() <= TOL * max(h * h, area) * big
    # a cell of the pixel, or one whose side is on its line
    num = d.image_of_cell_nums([lo, lo], [hi, hi], (res, res))
    assert (num >= 0).all()
    q = p[num]
    mid = lo + (np.arange(res) + 0.5) * ps
    reach = 0.5 * (h + ps) * (1 + 1e-9)
    assert (np.abs(q[..., 0] - mid[None, :]) <= reach).all() and (np.abs(q[..., 1] - mid[:, None]) <= reach).all()
