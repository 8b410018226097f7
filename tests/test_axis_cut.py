"""The cut of a cell to a pixel's line (axis_cut), compiled for the host, over
polygons of which a side lies on the line up to rounding.

A corner split into several vertices at one place, some of them outside by an
ulp, crosses the line four times and more.  The polygon is, bit for bit, what
cutting edge by edge into another buffer gives; where there is room for one more
vertex only, sides of length 1 and vertices off the line by at most 2^-52 leave
its area within 2^-52 a vertex of the exact one: ATOL = 1e-14 covers 40."""
import ctypes
import itertools
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ATOL = 1e-14
OWN = -1
ULP = 2.0 ** -52


@pytest.fixture(scope="module")
def axis_cut(tmp_path_factory):
    lib = str(tmp_path_factory.mktemp("axis_cut") / "axis_cut.so")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-w", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "sdot_b200", "csrc"), "-I" + os.path.join(cuda, "include"),
                    os.path.join(ROOT, "tests", "axis_cut_host.cpp"), "-o", lib], check=True)
    fn = ctypes.CDLL(lib).axis_cut_host
    P = ctypes.c_void_p
    fn.argtypes = [P, P, P, ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_double, ctypes.c_double, ctypes.c_int,
                   ctypes.c_int]

    def cut(poly, axis, c, s, more):
        # more: vertices that fit beside the polygon's own
        m = len(poly)
        cap = m + more
        x, y = np.full(cap + 2, 7e77), np.full(cap + 2, 7e77)
        ids = np.full(cap + 2, -99, np.int32)
        x[:m], y[:m], ids[:m] = poly[:, 0], poly[:, 1], np.arange(m)
        n = fn(x.ctypes.data, y.ctypes.data, ids.ctypes.data, m, cap, axis, c, s, OWN, cap)
        assert 0 <= n <= cap
        assert (x[cap:] == 7e77).all() and (y[cap:] == 7e77).all() and (ids[cap:] == -99).all()
        return np.stack([x[:n], y[:n]], 1), ids[:n]

    return cut


def edge_by_edge(poly, axis, c, s):
    out, ids = [], []
    m = len(poly)
    for k in range(m):
        a, b = poly[k], poly[(k + 1) % m]
        va, vb = s * (a[axis] - c), s * (b[axis] - c)
        if va >= 0:
            out.append(a)
            ids.append(k)
        if (va >= 0) != (vb >= 0):
            p = a + va / (va - vb) * (b - a)
            p[axis] = c
            out.append(p)
            ids.append(OWN if va >= 0 else k)
    return np.array(out).reshape(-1, 2), np.array(ids, int)


def area(p):
    if len(p) < 3:
        return 0.0
    q = p - p[0]
    return 0.5 * float(np.sum(q[:-1, 0] * q[1:, 1] - q[1:, 0] * q[:-1, 1]))


def changes(poly, axis, c, s):
    o = s * (poly[:, axis] - c) >= 0
    return int(np.sum(o != np.roll(o, -1)))


def turned(poly, axis, s):
    """The polygon with its side on y = 1 taken to x = 1 or the other sign."""
    p = poly.copy()
    if s > 0:
        p = 2.0 - p  # a half turn about (1, 1): the rest lies above the line
    if axis == 0:
        p = np.stack([p[:, 1], 2.0 - p[:, 0]], 1)  # a quarter turn clockwise about (1, 1)
    return p


@pytest.mark.parametrize("inside", [True, False])
@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("s", [-1.0, 1.0])
def test_side_on_the_line(axis_cut, axis, s, inside):
    # unit squares with up to six vertices on y = 1, split corners among them,
    # each an ulp in or out, from every starting vertex
    seen = set()
    for xs in ([1.0, 0.0], [1.0, 1.0, 0.0, 0.0], [1.0, 1.0, 0.6, 0.4, 0.0, 0.0], [1.0, 1.0, 1.0, 0.0, 0.0, 0.0]):
        for signs in itertools.product([-1, 0, 1], repeat=len(xs)):
            line = np.array([[x, 1.0 + d * ULP] for x, d in zip(xs, signs)])
            base = np.concatenate([[[0.0, 0.0], [1.0, 0.0]], line])
            for start in range(len(base)):
                p = turned(np.roll(base, -start, axis=0), axis, s)
                side = s if inside else -s
                seen.add(changes(p, axis, 1.0, side))
                want, wid = edge_by_edge(p, axis, 1.0, side)
                for more in (1, 4):
                    got, ids = axis_cut(p, axis, 1.0, side, more)
                    assert abs(area(got) - (1.0 if inside else 0.0)) <= ATOL, (xs, signs, start, more)
                    if more == 4 or changes(p, axis, 1.0, side) <= 2:
                        assert np.array_equal(got, want) and np.array_equal(ids, wid)
    assert {0, 2, 4, 6} <= seen


def test_line_through_the_middle(axis_cut):
    # any convex polygon: two changes at most, the same bits
    rng = np.random.default_rng(3)
    for _ in range(2000):
        m = int(rng.integers(3, 20))
        a = np.sort(rng.uniform(0, 2 * np.pi, m))
        p = np.stack([np.cos(a), np.sin(a)], 1)
        axis, c, s = int(rng.integers(2)), float(rng.uniform(-1.1, 1.1)), float(rng.choice([-1.0, 1.0]))
        got, ids = axis_cut(p, axis, c, s, 1)
        want, wid = edge_by_edge(p, axis, c, s)
        assert np.array_equal(got, want) and np.array_equal(ids, wid)
