"""The plain form's structured FP64 LDL^T (csrc/ldl64.cu) against dense numpy
solves of the same system, at the edges of its panels (32 columns, the split at
m and 2m), of its tiles and of its solve paths, and its hand-over to the
pivoted LU. Tolerance: both sides solve in FP64 with backward errors of a few
eps N; 1e-10 of the largest unknown covers systems of N = 400 by three orders."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-10


def wire(pkg, m):
    """A bent wire of m segments (m + 1 nodes) below the surface."""
    rng = np.random.default_rng(m)
    steps = rng.uniform(0.4, 1.0, (m, 3)) * np.where(np.arange(m)[:, None] % 2 == np.arange(3), 1.0, 0.0)
    nodes = np.concatenate([[[0.0, 0.0, -0.6]], [0.0, 0.0, -0.6] + np.cumsum(steps, axis=0)])
    return np.stack([pkg.populate_electrode(nodes[i], nodes[i + 1], 7e-3) for i in range(m)]), nodes


def dense_solution(pkg, e, img, nodes, s, kappa, inj):
    m, n = len(e), len(nodes)
    N = n + 2 * m
    zl, zt = np.zeros(m * m, np.complex128), np.zeros(m * m, np.complex128)
    gamma, ref_t = pkg.medium(s, kappa)
    assert pkg.calculate_impedances(zl, zt, e, gamma, s, 1.0, kappa) == 0
    assert pkg.impedances_images(zl, zt, e, img, gamma, s, 1.0, kappa, 1.0, ref_t) == 0
    wg = np.zeros(N * N, np.complex128)
    assert pkg.fill_incidence_imm(wg, e, nodes) == 0
    assert pkg.fill_impedance_imm(wg, zl, zt, m, n) == 0
    w = np.tril(wg.reshape(N, N).T)
    b = np.zeros(N, np.complex128)
    b[inj] = 1.0
    return np.linalg.solve(w + np.tril(w, -1).T, b)


@pytest.mark.parametrize("m", [1, 2, 10, 11, 20, 21, 22, 31, 32, 33, 64, 65, 106, 107, 129])
@pytest.mark.parametrize("graphs", [True, False])
def test_plain_plan_matches_dense_solve(gpu_pkg, m, graphs):
    """One CTA per sample up to N = 64 (m = 21), one-CTA solves up to N = 320
    (m = 106), panel launches above."""
    pkg = gpu_pkg
    e, nodes = wire(pkg, m)
    img = pkg.images(e)
    s = 8e4 + 2j * np.pi * np.array([1e3, 1e6])
    kappa = 0.01 + s * 12 * pkg.EPS0
    sol, info, _ = pkg.hem_sweep(e, img, nodes, s, kappa, inj_node=m // 2, graphs=graphs)
    assert not info.any()
    for k in range(2):
        assert rel_err(sol[k], dense_solution(pkg, e, img, nodes, s[k], kappa[k], m // 2)) < TOL


@pytest.mark.parametrize("ns", [1, 127, 128, 131])
def test_plain_plan_batches_agree(gpu_pkg, ns):
    """The panel launches' solve (up to 127 samples) and the one-CTA solve
    (from 128) of N = 358, and both panel CTA sizes, against single samples."""
    pkg = gpu_pkg
    e, nodes = wire(pkg, 119)
    img = pkg.images(e)
    s = 8e4 + 2j * np.pi * np.linspace(1e4, 5e6, ns)
    kappa = 0.002 + s * 8 * pkg.EPS0
    sol, info, _ = pkg.hem_sweep(e, img, nodes, s, kappa, max_batch=ns)
    assert not info.any()
    for k in {0, ns // 2, ns - 1}:
        alone, _, _ = pkg.hem_sweep(e, img, nodes, s[k:k + 1], kappa[k:k + 1])
        assert rel_err(sol[k], alone[0]) < TOL


@pytest.mark.parametrize("graphs", [True, False])
def test_samples_without_static_pivots_go_to_the_pivoted_lu(gpu_pkg, graphs):
    """s = 0 makes ZL zero: the static order meets zero pivots, the system of a
    tree of segments is still regular."""
    pkg = gpu_pkg
    e, nodes = wire(pkg, 40)
    img = pkg.images(e)
    s = np.array([0.0, 8e4 + 1e6j, 0.0])
    kappa = np.array([0.01 + 0j, 0.01 + 1e-4j, 0.02 + 0j])
    sol, info, _ = pkg.hem_sweep(e, img, nodes, s, kappa, inj_node=3, graphs=graphs)
    assert not info.any()
    for k in range(3):
        assert rel_err(sol[k], dense_solution(pkg, e, img, nodes, s[k], kappa[k], 3)) < TOL
    jobs = [{"electrodes": e, "images": img, "nodes": nodes, "s": s, "kappa": kappa, "inj_node": 3}]
    (got, binfo), = pkg.solve_batch(jobs, precision=pkg.PLAIN_FP64)
    assert not binfo.any()
    assert rel_err(got, sol) < TOL


def symmetric(rng, N):
    a = rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))
    return a + a.T + 2 * N * np.eye(N)


@pytest.mark.parametrize("m,n", [(1, 1), (15, 2), (16, 1), (40, 33), (110, 101)])
@pytest.mark.parametrize("kind", ["structured", "coupled", "zero pivots"])
def test_solve_immittance_of_any_symmetric_matrix(gpu_pkg, m, n, kind):
    """The structured elimination, a caller's matrix with a ZL/ZT coupling, and
    one whose impedance blocks have a zero diagonal (pivoted LU)."""
    pkg = gpu_pkg
    rng = np.random.default_rng(m + n)
    N = n + 2 * m
    w = symmetric(rng, N)
    if kind != "coupled":
        w[n:n + m, n + m:] = 0
        w[n + m:, n:n + m] = 0
    if kind == "zero pivots":
        w -= np.diag(np.diag(w))
        if m == 1:
            w[n, 0] = w[0, n] = 3.0
            w[n + 1, n + 1] = 2.0
    x = rng.standard_normal(N) + 1j * rng.standard_normal(N)
    b = w @ x
    lower = np.tril(w).T.ravel().copy()             # column-major, upper triangle unread
    got = b.copy()
    assert pkg.solve_immittance(lower, got, m, n) == 0
    assert rel_err(got, np.linalg.solve(w, b)) < 1e-9


@pytest.mark.parametrize("m,n", [(1, 1), (31, 3), (32, 33), (65, 40), (130, 7)])
@pytest.mark.parametrize("zero_diagonal", [False, True])
def test_yla_ytb_of_any_symmetric_blocks(gpu_pkg, m, n, zero_diagonal):
    pkg = gpu_pkg
    rng = np.random.default_rng(m * n)
    z = [symmetric(rng, m) for _ in range(2)]
    if zero_diagonal and m > 1:
        z[1] -= np.diag(np.diag(z[1]))
    rhs = [(rng.standard_normal((m, n)) + 0j) for _ in range(2)]
    zl, zt = (np.tril(v).T.ravel().copy() for v in z)
    a, b = (v.T.ravel().copy() for v in rhs)
    yla, ytb = np.zeros(m * n, np.complex128), np.zeros(m * n, np.complex128)
    assert pkg.calculate_yla_ytb(yla, ytb, zl, zt, a, b, m, n) == 0
    for got, inv, v, r in ((yla, zl, z[0], rhs[0]), (ytb, zt, z[1], rhs[1])):
        assert rel_err(got.reshape(n, m).T, np.linalg.solve(v, r)) < 1e-9
        assert rel_err(np.tril(inv.reshape(m, m).T), np.tril(np.linalg.inv(v))) < 1e-9


@pytest.mark.parametrize("m,n", [(1, 700), (32, 1100), (33, 290), (97, 80), (257, 40)])
def test_yla_ytb_of_one_to_eight_columns_per_cta(gpu_pkg, m, n):
    """Widths of the column tiles of the nodal solve, with a ragged last one."""
    test_yla_ytb_of_any_symmetric_blocks(gpu_pkg, m, n, False)


@pytest.mark.parametrize("m,ns", [(22, 1), (106, 38), (106, 39), (107, 19), (107, 20), (171, 3), (341, 2), (342, 2)])
def test_plain_plan_solves_on_clusters(gpu_pkg, m, ns):
    """The cluster solve and its limits: N = 1024 (m = 341), two waves of clusters up to N = 320, one above."""
    pkg = gpu_pkg
    e, nodes = wire(pkg, m)
    img = pkg.images(e)
    s = 8e4 + 2j * np.pi * np.linspace(1e3, 1e6, ns)
    kappa = 0.01 + s * 12 * pkg.EPS0
    sol, info, _ = pkg.hem_sweep(e, img, nodes, s, kappa, inj_node=m // 2, max_batch=ns)
    assert not info.any()
    for k in {0, ns - 1}:
        assert rel_err(sol[k], dense_solution(pkg, e, img, nodes, s[k], kappa[k], m // 2)) < TOL


def refined_solution(w, b):
    """Dense solve with the residual in extended precision."""
    x = np.linalg.solve(w, b).astype(np.clongdouble)
    wide = w.astype(np.clongdouble)
    for _ in range(4):
        x = x + np.linalg.solve(w, (b - wide @ x).astype(np.complex128))
    return x


@pytest.mark.parametrize("s", [1e-2, 1.0 + 10.0j, 1e2 + 1e2j, 8e4 + 1e3j, 8e4 + 1e6j])
@pytest.mark.parametrize("sigma", [1e-6, 1e-4, 1e-2])
@pytest.mark.parametrize("mesh", [2, 4])
def test_currents_and_potentials_each_match_extended_precision(gpu_pkg, s, sigma, mesh):
    """Potentials reach 1e4 V and more per ampere towards DC in resistive soil,
    where a longitudinal current follows from a difference of potentials that
    agree to 8 digits and more: the three blocks of the solution each against a
    solve refined in extended precision, through the plan and solve_immittance.
    Bound 1e-11 of the block's largest value: the solves' own 1e-15 or so and,
    between the plan's fill and the drop-ins', entries that differ by 1e-15 in a
    system whose impedance part has a condition number up to ~1e3."""
    pkg = gpu_pkg
    e, nodes = pkg.electrode_grid(mesh + 1, mesh + 1, 60.0, 60.0, 2, 2, 7e-3, -0.5)
    img, inj = pkg.images(e), 5
    m, n = len(e), len(nodes)
    N = n + 2 * m
    s = complex(s)
    kappa = sigma + s * 10 * pkg.EPS0
    zl, zt = np.zeros(m * m, np.complex128), np.zeros(m * m, np.complex128)
    gamma, ref_t = pkg.medium(s, kappa)
    assert pkg.calculate_impedances(zl, zt, e, gamma, s, 1.0, kappa) == 0
    assert pkg.impedances_images(zl, zt, e, img, gamma, s, 1.0, kappa, 1.0, ref_t) == 0
    wg = np.zeros(N * N, np.complex128)
    assert pkg.fill_incidence_imm(wg, e, nodes) == 0
    assert pkg.fill_impedance_imm(wg, zl, zt, m, n) == 0
    w = np.tril(wg.reshape(N, N).T)
    w = w + np.tril(w, -1).T
    x = np.zeros(N, np.complex128)
    x[inj] = 1.0
    want = refined_solution(w, x)
    assert pkg.solve_immittance(wg, x, m, n) == 0
    sol, info, _ = pkg.hem_sweep(e, img, nodes, np.array([s]), np.array([kappa]), inj_node=inj)
    assert not info.any()
    for part in (slice(0, n), slice(n, n + m), slice(n + m, N)):
        scale = np.abs(want[part]).max()
        assert np.abs(x[part] - want[part]).max() <= 1e-11 * scale
        assert np.abs(sol[0][part] - want[part]).max() <= 1e-11 * scale


@pytest.mark.parametrize("s", [1e-3, 0.31, 13.0])
@pytest.mark.parametrize("length,m,sigma", [(1300.0, 15, 1.5e-7), (5.6, 74, 3.8e-2), (5.7, 95, 4.3e-5), (4.4, 62, 0.11),
                                            (110.0, 81, 1.3e-3), (60.0, 130, 1e-3)])
def test_refinement_goes_on_until_rounding(gpu_pkg, length, m, sigma, s):
    """Real s towards DC: ZL is so small that the static order loses the ground
    impedances' digits and refinement contracts by 1e-5 to 1e-3 only. Every
    block of the plan's and solve_immittance's solution (one CTA per sample,
    clusters, panels) against a solve refined in extended precision: a few N eps,
    2e-13 for N up to 391."""
    pkg = gpu_pkg
    e, nodes = pkg.segment_electrode([0.0, 0.0, -0.5], [length, 0.0, -0.5], m, 5e-3)
    img, inj, n = pkg.images(e), m // 3, m + 1
    N = n + 2 * m
    s = complex(s)
    kappa = sigma + s * 10 * pkg.EPS0
    zl, zt = np.zeros(m * m, np.complex128), np.zeros(m * m, np.complex128)
    gamma, ref_t = pkg.medium(s, kappa)
    assert pkg.calculate_impedances(zl, zt, e, gamma, s, 1.0, kappa) == 0
    assert pkg.impedances_images(zl, zt, e, img, gamma, s, 1.0, kappa, 1.0, ref_t) == 0
    wg = np.zeros(N * N, np.complex128)
    assert pkg.fill_incidence_imm(wg, e, nodes) == 0
    assert pkg.fill_impedance_imm(wg, zl, zt, m, n) == 0
    w = np.tril(wg.reshape(N, N).T)
    w = w + np.tril(w, -1).T
    x = np.zeros(N, np.complex128)
    x[inj] = 1.0
    want = refined_solution(w, x)
    assert pkg.solve_immittance(wg, x, m, n) == 0
    sol, info, _ = pkg.hem_sweep(e, img, nodes, np.array([s]), np.array([kappa]), inj_node=inj)
    assert not info.any()
    for part in (slice(0, n), slice(n, n + m), slice(n + m, N)):
        scale = np.abs(want[part]).max()
        assert np.abs(x[part] - want[part]).max() <= 2e-13 * scale
        assert np.abs(sol[0][part] - want[part]).max() <= 2e-13 * scale


@pytest.mark.parametrize("m", [15, 74, 130])
@pytest.mark.parametrize("kind", ["s = 0", "sub-hertz", "both and usual ones"])
@pytest.mark.parametrize("graphs", [True, False])
def test_hard_samples_are_solved_side_by_side(gpu_pkg, m, kind, graphs):
    """Samples that need more corrections than a pass makes, or the pivoted LU, go through those together, in plans (two
    passes, the second shorter) and in a grid batch: launches that do not grow with their number (a LU takes four per 32
    unknowns and two sweeps of two; the structured solve four a correction, up to 32 unknowns a launch in its sweeps),
    and every sample against the same solved alone."""
    pkg = gpu_pkg
    e, nodes = pkg.segment_electrode([0.0, 0.0, -0.5], [0.08 * m, 0.0, -0.5], m, 5e-3)
    img, ns = pkg.images(e), 60
    N = 3 * m + 1
    hard = 2j * np.pi * np.logspace(-2, 0, ns)
    s = {"s = 0": np.zeros(ns, np.complex128), "sub-hertz": hard,
         "both and usual ones": np.where(np.arange(ns) % 3 == 0, 0.0, np.where(np.arange(ns) % 3 == 1, hard, 8e4 + 1e5j))}[kind]
    kappa = np.full(ns, 1e-4 + 0j)
    plan = pkg.Plan(e, img, nodes, pkg.PLAIN_FP64, 40, graphs)
    try:
        plan.run(s, kappa, inj_node=2)                      # graphs built
        before = pkg.launch_count()
        sol, info, _ = plan.run(s, kappa, inj_node=2)
        launches = pkg.launch_count() - before
        assert not info.any()
        panels = (N + 31) // 32 + 2
        assert launches <= 2 * (60 + panels * (2 + 14 * 2 + 2 + 8))
        for k in (0, 1, 2, 39, 40, 59):
            alone, info, _ = plan.run(s[k:k + 1], kappa[k:k + 1], inj_node=2)
            assert not info.any()
            for part in (slice(0, m + 1), slice(m + 1, 2 * m + 1), slice(2 * m + 1, N)):
                assert np.abs(sol[k][part] - alone[0][part]).max() <= 2e-13 * np.abs(alone[0][part]).max()
    finally:
        plan.close()
    if graphs:
        jobs = [{"electrodes": e, "images": img, "nodes": nodes, "s": s, "kappa": kappa, "inj_node": 2}]
        (got, info), = pkg.solve_batch(jobs, precision=pkg.PLAIN_FP64)
        assert not info.any()
        for part in (slice(0, m + 1), slice(m + 1, 2 * m + 1), slice(2 * m + 1, N)):
            scale = np.abs(sol[:, part]).max(axis=1)
            assert (np.abs(got[:, part] - sol[:, part]).max(axis=1) <= 2e-13 * scale).all()
