"""A wait of the kernels whose blocks meet at barriers (sort, tree, conjugate
gradients) that is given up ends in an error status: a library whose waits all
give up at once (SDOT_BARRIER_SPINS=0) sorts nothing and builds no tree, and every
call says so, reads and writes in range, and leaves the device usable."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = r"""
import sys
import numpy as np
import torch
sys.path.insert(0, {root!r})
from sdot_b200._lib import SDOT_ITER_CAP, SdotError
from sdot_b200.power_diagram import PowerDiagram

def lost(f):
    try:
        f()
    except SdotError as e:
        assert e.status == SDOT_ITER_CAP and "given up" in str(e), str(e)
    else:
        raise AssertionError("no error")

for dim in (2, 3):
    for n in (1, 700, 20000):
        p = np.random.default_rng(n).random((n, dim))
        d = PowerDiagram(p, np.zeros(n))
        d.add_box_shape(np.zeros(dim), np.ones(dim))
        # twice: the tree is built again
        for _ in range(2):
            lost(d.integrals)
            lost(d.neighbors)
        lost(lambda: d.solve_weights(np.full(n, 1 / n)))
        d.set_weights(np.full(n, 1e-6))
        lost(d.der_integrals_wrt_weights)
        if dim == 2:
            lost(d.der_centroids_and_integrals_wrt_weight_and_positions)
            lost(lambda: d.image_integrals([0, 0], [1, 1], (8, 8)))
            lost(lambda: d.image_of_cell_nums([0, 0], [1, 1], (8, 8)))
torch.cuda.synchronize()
assert float(torch.ones(1000, device="cuda").sum()) == 1000
print("all given up")
"""


@pytest.fixture(scope="module")
def no_wait_lib(cuda_ok):
    from sdot_b200 import build

    build.build()
    lib = os.path.join(build.HERE, "libsdot_b200_no_wait.so")
    if not os.path.exists(lib) or os.path.getmtime(lib) < os.path.getmtime(build.LIB):
        build.build(force=True, extra=["-DSDOT_BARRIER_SPINS=0"], lib=lib)
    return lib


def test_every_wait_given_up(no_wait_lib):
    r = subprocess.run([sys.executable, "-c", CODE.format(root=ROOT)], env=dict(os.environ, SDOT_B200_LIB=no_wait_lib),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "all given up" in r.stdout
