"""Regular lattices of Diracs: the corners of the cells are several vertices at
one place, of which a cut may find some outside by an ulp here and there.  Every
cell is a square; TOL as in test_gpu_lattice_pixels.py.  Warps of their own up to
6,000 Diracs (77 a side), 12 and 32 cells a warp above."""
import numpy as np
import pytest

from sdot_b200.power_diagram import PowerDiagram
from tests.test_gpu_lattice_pixels import BOXES, TOL, lattice

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo,hi", BOXES)
@pytest.mark.parametrize("m", list(range(10, 130, 3)) + [200, 300, 362])
def test_squares(gpu_lib, m, lo, hi):
    p, _, h = lattice(m, lo, hi)
    d = PowerDiagram(p, np.zeros(m * m))
    d.add_box_shape([lo, lo], [hi, hi])
    c, mass = d.centroids(with_masses=True)
    assert np.abs(mass - h * h).max() <= TOL * h * h
    assert np.abs(c - p).max() <= TOL * max(abs(lo), abs(hi))
