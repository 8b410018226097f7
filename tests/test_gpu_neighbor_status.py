"""The status of neighbour lists and position derivatives is that of the walk that
made them: not of an earlier evaluation, and not lost in a call that makes no
evaluation."""
import numpy as np
import pytest

from sdot_b200._lib import SDOT_CAPACITY, SdotError
from sdot_b200.power_diagram import PowerDiagram
from tests.test_gpu_cell3d_capacity import diagram as diagram3d
from tests.test_gpu_cell3d_capacity import sphere
from tests.test_gpu_derpos_rows import ring

pytestmark = pytest.mark.gpu


def circle(m):
    """One Dirac inside m others at one distance: a cell of m edges."""
    a = 2 * np.pi * (np.arange(m) + np.random.default_rng(m).uniform(-0.1, 0.1, m)) / m
    return np.concatenate([0.5 + 0.3 * np.stack([np.cos(a), np.sin(a)], 1), [[0.5, 0.5]]])


def diagram(p):
    g = PowerDiagram(p, np.zeros(len(p)))
    g.add_box_shape([0, 0], [1, 1])
    return g


def derivatives(g):
    return g.der_centroids_and_integrals_wrt_weight_and_positions()


def fails(f):
    with pytest.raises(SdotError) as e:
        f()
    assert e.value.status == SDOT_CAPACITY


def good():
    return np.random.default_rng(11).random((500, 2))


def check_good(g):
    """The outputs of a fresh context."""
    g.set_positions_and_weights(good(), np.zeros(500))
    f = diagram(good())
    for a, b in zip(derivatives(g), derivatives(f)):
        assert np.array_equal(a, b)
    for a, b in zip(g.neighbors(), f.neighbors()):
        assert np.array_equal(a, b)
    assert np.array_equal(g.integrals(), f.integrals())


@pytest.mark.parametrize("first", ["integrals", "derivatives", "neighbors"])
@pytest.mark.parametrize("m", [1100])
def test_cells_past_the_last_tier(gpu_lib, m, first):
    # a first call of each kind, then the others, then other Diracs
    g = diagram(circle(m))
    calls = {"integrals": g.integrals, "derivatives": lambda: derivatives(g), "neighbors": g.neighbors}
    fails(calls.pop(first))
    for f in calls.values():
        fails(f)
        fails(f)
    check_good(g)


def test_derivatives_past_their_own_capacity(gpu_lib):
    # 65 edges: the walk is sound, its other outputs are there
    g = diagram(ring(65))
    fails(lambda: derivatives(g))
    off, ids = g.neighbors()
    assert off[66] - off[65] == 65
    assert abs(g.integrals().sum() - 1) < 1e-12
    check_good(g)


def test_good_lists_beside_a_failed_evaluation(gpu_lib):
    # the status of one is not the other's, in either order
    g = diagram(circle(1100))
    fails(g.integrals)
    g.set_positions_and_weights(good(), np.zeros(500))
    derivatives(g)
    g.neighbors()
    g.set_positions_and_weights(circle(1100), np.zeros(1101))
    fails(g.neighbors)
    g.set_positions_and_weights(good(), np.zeros(500))
    assert abs(g.integrals().sum() - 1) < 1e-12


def test_polyhedra_past_the_last_pass(gpu_lib):
    g = diagram3d(sphere(300))
    fails(g.neighbors)
    p = np.random.default_rng(12).random((300, 3))
    g.set_positions_and_weights(p, np.zeros(300))
    for a, b in zip(g.neighbors(), diagram3d(p).neighbors()):
        assert np.array_equal(a, b)
