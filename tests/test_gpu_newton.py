"""Newton on the weights on the GPU vs the Newton oracle (compiled reference
CSR + a direct sparse solve, oracle/newton.py).

Both solves run to a relative mass error of 1e-12 from the same start; the
gauge fix pins the weight of Dirac 0, so the weights themselves are compared:
|w_gpu - w_ref| <= 1e-10 max |w_ref| (the round-off of a 1e-12 mass error
amplified by the inverse Hessian, whose norm grows like n).
"""
import numpy as np
import pytest

from oracle import newton
from sdot_b200 import workloads

pytestmark = pytest.mark.gpu

W_RTOL = 1e-10


def solve_pair(ref_oracle, p, w0, target, radial_func="unit", image=None, rule="damped", tol=1e-12):
    from sdot_b200.power_diagram import PowerDiagram

    gpu = PowerDiagram(p, w0, radial_func=radial_func)
    ref = ref_oracle.RefPowerDiagram(p, w0, radial_func=radial_func)
    if image is not None:
        gpu.set_image_density(image)
        ref.set_image_density(image)
    else:
        gpu.add_box_shape([0.0, 0.0], [1.0, 1.0])
        ref.add_box_shape([0.0, 0.0], [1.0, 1.0])
    rep = gpu.solve_weights(target, rel_mass_tol=tol, damping=(rule == "damped"))
    w_r, rep_r = newton.solve(ref, target, w0, tol=tol, rule=rule, ball_cut=(radial_func != "unit"))
    assert rep_r["converged"]
    return gpu, gpu.get_weights(), w_r, rep, rep_r


def check_weights(w_g, w_r):
    err = np.abs(w_g - w_r).max() / np.abs(w_r).max()
    assert err <= W_RTOL, f"weights differ by {err:.3e} of max |w|"


@pytest.mark.parametrize("rule", ["damped", "reference"])
def test_newton_config1(gpu_lib, ref_oracle, rule):
    c = workloads.config1()
    n = len(c["weights"])
    gpu, w_g, w_r, rep, rep_r = solve_pair(ref_oracle, c["positions"], c["weights"], np.full(n, 1.0 / n), rule=rule)
    assert rep["max_rel_mass_error"] <= 1e-12
    check_weights(w_g, w_r)
    m = gpu.integrals()
    assert np.abs(m * n - 1).max() <= 1e-12


def test_newton_clustered(gpu_lib, ref_oracle):
    rng = np.random.default_rng(11)
    n = 5000
    p = np.concatenate([rng.random((n // 2, 2)), workloads.clustered_points(n - n // 2, 2, rng)])
    # tight clusters: the reachable relative mass error is ~7e-12 (CPU oracle)
    gpu, w_g, w_r, rep, rep_r = solve_pair(ref_oracle, p, np.zeros(n), np.full(n, 1.0 / n), tol=2e-11)
    check_weights(w_g, w_r)


def test_newton_disc_clip_partial(gpu_lib, ref_oracle):
    # partial transport: cells clipped by the disc of radius sqrt(w_i), total
    # target 0.8 of the unit box; no gauge fix (the arcs make H regular)
    rng = np.random.default_rng(12)
    n = 2000
    p = rng.random((n, 2))
    w0 = np.full(n, (0.5 / np.sqrt(n)) ** 2)
    gpu, w_g, w_r, rep, rep_r = solve_pair(ref_oracle, p, w0, np.full(n, 0.8 / n), radial_func="in_ball_w05")
    check_weights(w_g, w_r)


def test_newton_image_density(gpu_lib, ref_oracle):
    rng = np.random.default_rng(13)
    n = 3000
    p = rng.random((n, 2))
    img = workloads.c3_image(res=64)
    gpu, w_g, w_r, rep, rep_r = solve_pair(ref_oracle, p, np.zeros(n), np.full(n, 0.8 / n), image=img)
    check_weights(w_g, w_r)


def test_optimal_transport_facade_collinear_pairs(gpu_lib, ref_oracle):
    # the reference's example: 20 pairs of close Diracs on the line y = 0.5
    # (every cell a vertical strip), default unit box and equal masses
    from sdot_b200.optimal_transport import OptimalTransport

    xs = np.linspace(0, 1 - 1e-3, 20)
    pos = np.array([[x + d, 0.5] for x in xs for d in (0.0, 1e-3)])
    ot = OptimalTransport(pos)
    ot.adjust_weights()
    w_g = ot.get_weights()
    m = ot.get_integrals()
    assert np.abs(m * 40 - 1).max() <= 1e-10
    ref = ref_oracle.RefPowerDiagram(pos, np.zeros(40))
    ref.add_box_shape([0.0, 0.0], [1.0, 1.0])
    w_r, _ = newton.solve(ref, np.full(40, 1 / 40), np.zeros(40), tol=1e-10)
    assert np.abs(w_g - w_r).max() <= 1e-9 * np.abs(w_r).max()


def test_void_start_rejected_by_damped_newton(gpu_lib):
    from sdot_b200._lib import SDOT_VOID_CELL, SdotError
    from sdot_b200.power_diagram import PowerDiagram

    c = workloads.config2(n=20_000)
    g = PowerDiagram(c["positions"], c["weights"])
    g.add_box_shape([0.0, 0.0], [1.0, 1.0])
    assert (g.integrals() == 0).any()
    with pytest.raises(SdotError) as e:
        g.solve_weights(np.full(20_000, 1 / 20_000))
    assert e.value.status == SDOT_VOID_CELL


def test_csr_solve_matches_direct_solve(gpu_lib, ref_oracle):
    # the linear step alone: the reference CSR of C1 with the gauge fix,
    # device conjugate gradients vs a direct sparse solve
    import scipy.sparse as sp
    import scipy.sparse.linalg as spla

    from sdot_b200.power_diagram import csr_solve

    c = workloads.config1()
    n = len(c["weights"])
    ref = ref_oracle.RefPowerDiagram(c["positions"], c["weights"])
    ref.add_box_shape([0.0, 0.0], [1.0, 1.0])
    err, off, col, val, m = ref.der_integrals_wrt_weights()
    b = m - 1.0 / n + np.random.default_rng(3).normal(0, 1e-6, n)
    x, it, res = csr_solve(off, col, val, b, gauge_fix=True, rel_tol=1e-13)
    v2 = val.copy()
    v2[0] *= 2
    x_ref = spla.spsolve(sp.csr_matrix((v2, col, off), shape=(n, n)).tocsc(), b)
    assert res <= 1e-13
    assert np.abs(x - x_ref).max() <= 1e-8 * np.abs(x_ref).max()


def test_multilevel_and_jacobi_give_the_same_weights(gpu_lib):
    # the preconditioner changes the CG path, not the Newton solution
    from sdot_b200.power_diagram import PowerDiagram

    c = workloads.config1()
    n = len(c["weights"])
    out = {}
    for pc in ("multilevel", "jacobi"):
        g = PowerDiagram(c["positions"], np.zeros(n))
        g.add_box_shape([0, 0], [1, 1])
        rep = g.solve_weights(c["target"], rel_mass_tol=1e-11, preconditioner=pc)
        out[pc] = (g.get_weights(), rep)
    (wm, rm), (wj, rj) = out["multilevel"], out["jacobi"]
    assert rm["pcg_levels"] >= 2 and rj["pcg_levels"] == 0
    assert rm["pcg_iterations"] * 3 < rj["pcg_iterations"]
    assert np.abs(wm - wj).max() <= 1e-9 * np.abs(wj).max()


def test_multilevel_newton_clamped_clusters(gpu_lib):
    # Diracs clamped onto the box edges (the 1M clustered workload's
    # definition, here at 300k): sliver cells of mass ~1e-11 at w = 0, where
    # Jacobi-preconditioned CG stagnates.  Clamping also makes pairs of Diracs
    # on an edge 4e-8 apart, whose shared face FP64 cannot place finely
    # enough for 1e-8: the compiled reference with a direct solve stalls at a
    # relative mass error of 1.5e-6 on this input, so the bound is 1e-5.
    from sdot_b200.power_diagram import PowerDiagram

    c = workloads.config2(n=300_000)
    n = len(c["weights"])
    g = PowerDiagram(c["positions"], np.zeros(n))
    g.add_box_shape([0, 0], [1, 1])
    rep = g.solve_weights(c["target"], rel_mass_tol=1e-5)
    m = g.integrals()
    assert np.max(np.abs(m - c["target"]) / c["target"]) <= 1e-5
    assert rep["pcg_levels"] >= 4


def test_multilevel_newton_mirrored_clusters(gpu_lib):
    # the same mix with the clustered Diracs mirrored at the box faces (no
    # near-coincident pairs): 1e-8 from w = 0
    from sdot_b200.power_diagram import PowerDiagram

    rng = np.random.default_rng(52)
    n = 300_000
    p = np.concatenate([rng.random((n // 2, 2)), workloads.clustered_points(n - n // 2, 2, rng, boundary="reflect")])
    g = PowerDiagram(p, np.zeros(n))
    g.add_box_shape([0, 0], [1, 1])
    t = np.full(n, 1.0 / n)
    rep = g.solve_weights(t, rel_mass_tol=1e-8)
    m = g.integrals()
    assert np.max(np.abs(m - t) / t) <= 1e-8
    assert rep["pcg_levels"] >= 4


# ---- FP32 PCG with FP64 iterative refinement (linear_solver="fp32_refined"):
# the residuals and the weights stay FP64, so the solve reaches the same
# tolerance and Newton the same weights as with the FP64 PCG
def solve_gpu(p, w0, target, linear_solver, tol, radial_func="unit", image=None):
    from sdot_b200.power_diagram import PowerDiagram

    g = PowerDiagram(p, w0, radial_func=radial_func)
    if image is not None:
        g.set_image_density(image)
    else:
        g.add_box_shape(np.zeros(p.shape[1]), np.ones(p.shape[1]))
    rep = g.solve_weights(target, rel_mass_tol=tol, linear_solver=linear_solver)
    return g, g.get_weights(), rep


# The Newton iterates of the two linear solvers differ by rounding, and 1e-12
# is at the FP64 floor of C1's masses (the damped search may find no further
# decrease just above it), so the refined solves run to 1e-11 and their
# weights are held to 1e-9 of max |w| against the oracle's at 1e-12.
W_RTOL_REFINED = 1e-9


def test_refined_newton_config1_vs_oracle(gpu_lib, ref_oracle):
    c = workloads.config1()
    n = len(c["weights"])
    t = np.full(n, 1.0 / n)
    g, w_g, rep = solve_gpu(c["positions"], c["weights"], t, "fp32_refined", 1e-11)
    ref = ref_oracle.RefPowerDiagram(c["positions"], c["weights"])
    ref.add_box_shape([0.0, 0.0], [1.0, 1.0])
    w_r, rep_r = newton.solve(ref, t, c["weights"], tol=1e-12)
    assert rep["max_rel_mass_error"] <= 1e-11
    assert np.abs(w_g - w_r).max() <= W_RTOL_REFINED * np.abs(w_r).max()


def test_refined_csr_solve_matches_fp64(gpu_lib):
    # one linear solve: refined vs FP64 PCG on the same right-hand side, both
    # to a relative residual of 1e-12 (through the Newton step of C1 at w = 0)
    c = workloads.config1()
    n = len(c["weights"])
    ws = {}
    for ls in ("fp64", "fp32_refined"):
        g, w, rep = solve_gpu(c["positions"], np.zeros(n), c["target"], ls, 1e-11)
        ws[ls] = (w, rep)
    assert np.abs(ws["fp64"][0] - ws["fp32_refined"][0]).max() <= 1e-9 * np.abs(ws["fp64"][0]).max()
    assert ws["fp32_refined"][1]["iterations"] <= ws["fp64"][1]["iterations"] + 1


def test_refined_newton_disc_clip_image(gpu_lib, ref_oracle):
    c = workloads.config3(n=4000, res=64)
    n = len(c["weights"])
    g, w_g, rep = solve_gpu(c["positions"], c["weights"], c["target"], "fp32_refined", 1e-11,
                            radial_func="in_ball_w05", image=c["image"])
    ref = ref_oracle.RefPowerDiagram(c["positions"], c["weights"], radial_func="in_ball_w05")
    ref.set_image_density(c["image"])
    w_r, rep_r = newton.solve(ref, c["target"], c["weights"], tol=1e-12, ball_cut=True)
    assert rep_r["converged"]
    assert rep["max_rel_mass_error"] <= 1e-11
    # with the disc clip there is no gauge fix: a uniform shift of the weights
    # changes the masses only through the short arcs, so a 1e-11 mass error
    # leaves the weights free along it; the weights agree once that shift is
    # removed, and the shift itself is small
    d = w_g - w_r
    assert np.abs(d - d.mean()).max() <= 1e-10 * np.abs(w_r).max()
    assert abs(d.mean()) <= 1e-7 * np.abs(w_r).max()


def test_refined_newton_mirrored_clusters(gpu_lib):
    rng = np.random.default_rng(53)
    n = 300_000
    p = np.concatenate([rng.random((n // 2, 2)), workloads.clustered_points(n - n // 2, 2, rng, boundary="reflect")])
    t = np.full(n, 1.0 / n)
    g, w, rep = solve_gpu(p, np.zeros(n), t, "fp32_refined", 1e-8)
    m = g.integrals()
    assert np.max(np.abs(m - t) / t) <= 1e-8


def test_refined_newton_3d(gpu_lib):
    from sdot_b200.power_diagram import PowerDiagram

    c = workloads.config4(n=20_000)
    n = len(c["weights"])
    out = {}
    for ls in ("fp64", "fp32_refined"):
        g = PowerDiagram(c["positions"], c["weights"])
        g.add_box_shape([0, 0, 0], [1, 1, 1])
        g.set_polynomial_density(c["density"])
        g.solve_weights(c["target"], rel_mass_tol=1e-10, linear_solver=ls)
        out[ls] = g.get_weights()
    assert np.abs(out["fp64"] - out["fp32_refined"]).max() <= 1e-8 * np.abs(out["fp64"]).max()


@pytest.mark.parametrize("dim,n", [(2, 49), (2, 192), (2, 193), (2, 1025), (2, 2048), (2, 16390), (2, 38000), (3, 50),
                                   (3, 777), (3, 4100)])
def test_multilevel_solve_sizes(gpu_lib, dim, n):
    # the one-kernel multilevel solve where its levels and blocks change: the
    # smallest size it takes (49 rows), one and two levels, levels around the
    # largest that one block does alone, one row more or less than full blocks
    # and aggregates, more rows than one per thread of the grid.  The Newton
    # solution does not depend on the preconditioner: the bound of
    # test_multilevel_and_jacobi_give_the_same_weights
    from sdot_b200.power_diagram import PowerDiagram

    p = np.random.default_rng(5300 + n).random((n, dim))
    w = {}
    for pc, ls in (("jacobi", "fp64"), ("multilevel", "fp64"), ("multilevel", "fp32_refined")):
        g = PowerDiagram(p, np.zeros(n))
        g.add_box_shape(np.zeros(dim), np.ones(dim))
        rep = g.solve_weights(np.full(n, 1.0 / n), rel_mass_tol=1e-11, preconditioner=pc, linear_solver=ls)
        assert (rep["pcg_levels"] > 0) == (pc == "multilevel")
        w[pc, ls] = g.get_weights()
    ref = w["jacobi", "fp64"]
    for x in w.values():
        assert np.abs(x - ref).max() <= 1e-9 * np.abs(ref).max()


@pytest.mark.parametrize("n", [400_001, 401_409])
def test_multilevel_solve_larger_blocks(gpu_lib, n):
    # more than 400,000 rows: blocks of 512 threads, a row more than the line
    # and a ragged last block; the solved cells have their target masses
    from sdot_b200.power_diagram import PowerDiagram

    p = np.random.default_rng(5400 + n).random((n, 2))
    g = PowerDiagram(p, np.zeros(n))
    g.add_box_shape(np.zeros(2), np.ones(2))
    rep = g.solve_weights(np.full(n, 1.0 / n), rel_mass_tol=1e-8)
    assert rep["status"] == 0 and rep["pcg_levels"] > 0
    assert np.abs(g.integrals() * n - 1).max() <= 1e-8
