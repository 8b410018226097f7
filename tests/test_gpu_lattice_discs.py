"""Discs in the cells of regular lattices, whose corners are several vertices at
one place: a disc inside its cell is whole, one around it leaves the cell, and one
that reaches past the sides leaves no arc of a full turn in the slivers that a
pixel's line may cut off there.

Areas of a disc and of a square; TOL as in test_gpu_lattice_pixels.py (a disc's
own area, pi r^2, is exact to a few ulp)."""
import numpy as np
import pytest

from sdot_b200.power_diagram import PowerDiagram
from tests.test_gpu_lattice_pixels import BOXES, SIZES, TOL, lattice

pytestmark = pytest.mark.gpu


def share(rho):
    """Area of a disc of radius rho in a unit square about its centre."""
    if rho <= 0.5:
        return np.pi * rho * rho
    if rho * rho >= 0.5:
        return 1.0
    return np.pi * rho * rho - 4 * (rho * rho * np.arccos(0.5 / rho) - 0.5 * np.sqrt(rho * rho - 0.25))


def diagram(m, lo, hi, rho):
    p, order, h = lattice(m, lo, hi)
    return PowerDiagram(p, np.full(m * m, (rho * h) ** 2), radial_func="in_ball_w05"), h


@pytest.mark.parametrize("rho", [0.4, 0.55, 0.6, 0.7, 2.0])
@pytest.mark.parametrize("m,res", SIZES)
def test_discs_over_pixels(gpu_lib, m, res, rho):
    d, h = diagram(m, 0.1, 0.8, rho)
    d.set_image_density(np.ones((res, res)), [0.1, 0.1], [0.8, 0.8])
    assert np.abs(d.integrals() - share(rho) * h * h).max() <= TOL * h * h


@pytest.mark.parametrize("rho", [0.4, 0.6, 2.0])
@pytest.mark.parametrize("lo,hi", BOXES)
@pytest.mark.parametrize("m", [10, 49, 64, 97, 130, 200])
def test_discs_in_a_box(gpu_lib, m, lo, hi, rho):
    d, h = diagram(m, lo, hi, rho)
    d.add_box_shape([lo, lo], [hi, hi])
    assert np.abs(d.integrals() - share(rho) * h * h).max() <= TOL * h * h
    res = 2 * m + 1
    img = d.image_integrals([lo, lo], [hi, hi], (res, res))[..., 2]
    assert abs(img.sum() - m * m * share(rho) * h * h) <= TOL * m * m * h * h


@pytest.mark.parametrize("m", [20, 78, 129])
def test_discs_in_a_periodic_box(gpu_lib, m):
    d, h = diagram(m, 0.0, 1.0, 0.447)
    d.add_box_shape([0, 0], [1, 1])
    d.set_translations([[i, j] for i in (-1, 0, 1) for j in (-1, 0, 1) if i or j])
    assert np.abs(d.integrals() - share(0.447) * h * h).max() <= TOL * h * h


def test_discs_and_a_shape_of_no_width(gpu_lib):
    # the second shape holds no disc, whichever side of it a centre lies on
    rng = np.random.default_rng(5)
    p, w = rng.random((400, 2)), 0.25 / 400 * rng.uniform(0.3, 3.0, 400)
    one, two = [PowerDiagram(p, w, radial_func="in_ball_w05") for _ in range(2)]
    for d in (one, two):
        d.add_box_shape([0, 0], [1, 1], 0.5)
    two.add_box_shape([0.5, 0], [0.5, 1], 1.0)
    assert np.abs(two.integrals() - one.integrals()).max() <= TOL / 400
