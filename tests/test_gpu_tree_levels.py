"""The device tree and its sort at sizes around their blocks (512 pairs, 148
blocks), leaf sizes and depths: every Dirac in exactly one cell, neighbour lists
and masses those of the C restatement (oracle/port.py; bounds of the 2D parity
tests), new weights like a fresh diagram's (bit for bit: same tree, same walk)."""
import numpy as np
import pytest

from oracle import port
from sdot_b200.power_diagram import PowerDiagram
from tests.test_gpu_parity_2d import check_all

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,leaf", [(1, 11), (11, 11), (12, 11), (511, 1), (512, 11), (513, 11), (1025, 40), (9000, 3)])
def test_sizes_and_leaves(gpu_lib, n, leaf):
    rng = np.random.default_rng(8500 + n)
    p, w = rng.random((n, 2)), rng.uniform(-0.3, 0.3, n) / n
    g, r = PowerDiagram(p, w, max_diracs_per_cell=leaf), port.PortPowerDiagram(p, w)
    for d in (g, r):
        d.add_box_shape([0.0, 0.0], [1.0, 1.0])
    check_all(g, r, n, rtol_hess=1e-11)


@pytest.mark.parametrize("dim,n", [(2, 75_777), (2, 151_553), (2, 400_001), (3, 76_000)])
def test_many_blocks_and_new_weights(gpu_lib, dim, n):
    rng = np.random.default_rng(8600 + n)
    p = rng.random((n, dim))
    p[: n // 3] = 0.25 + 1e-4 * rng.random((n // 3, dim))  # deep levels
    g = PowerDiagram(p, np.zeros(n))
    g.add_box_shape(np.zeros(dim), np.ones(dim))
    assert abs(g.integrals().sum() - 1.0) < 1e-11
    w = rng.uniform(-1e-12, 1e-12, n)
    g.set_weights(w)
    f = PowerDiagram(p, w)
    f.add_box_shape(np.zeros(dim), np.ones(dim))
    for a, b in zip(g.der_integrals_wrt_weights(), f.der_integrals_wrt_weights()):
        assert np.array_equal(a, b)
