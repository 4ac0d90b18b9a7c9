"""GPU parity of the post-processing path (src/electrode.c:434-668 and the
closed-form mHEM ground potential of examples/visacro57emc01.c:406-430):
the four drop-ins and the three batched entry points against the reference's
own outputs (tests/golden/fields.npz, written by tests/golden/make_golden.py)
and against the oracle at tight cubature tolerance.

Tolerance: 1e-9 of the largest magnitude of each compared vector (the GPU
rules integrate to ~1e-12; the fixtures were made at 1e-11, the nested path
voltage at 1e-10, and path voltages are compared at 1e-8)."""
import numpy as np
import pytest

from conftest import golden

pytestmark = pytest.mark.gpu

TOL = 1e-9


def _close(got, want, axis=None):
    got = np.asarray(got)
    want = np.asarray(want)
    scale = np.max(np.abs(want), axis=axis, keepdims=axis is not None)
    err = np.abs(got - want) / np.maximum(scale, 1e-300)
    return float(np.max(err))


def _field_case():
    gd = golden("fields.npz")
    return {k: gd[k] for k in gd.files}


def test_fields_batch_matches_reference_fixture(gpu_pkg):
    pkg = gpu_pkg
    d = _field_case()
    before = pkg.launch_count()
    out = pkg.fields_batch(d["points"], d["elec"], d["il"], d["it"], d["gamma"], d["kappa"])
    assert pkg.launch_count() > before
    assert out["status"] == 0
    s = d["s"][:, None, None, None]
    full = out["efield"] - s * out["vecpot"]
    assert _close(out["pot"], d["pot"], axis=(1, 2)) <= TOL
    assert _close(out["vecpot"], d["vecpot"], axis=(1, 2, 3)) <= TOL
    assert _close(full, d["efield"], axis=(1, 2, 3)) <= TOL
    # s = 0 and a nonzero ve: the reference adds the conservative part to ve
    assert _close(out["efield"] + d["ve0"], d["efield_s0"], axis=(1, 2, 3)) <= TOL


def test_dropins_match_reference_fixture(gpu_pkg):
    pkg = gpu_pkg
    d = _field_case()
    e, pts = d["elec"], d["points"]
    for k in (0, 2):
        for r in range(d["il"].shape[1]):
            for p in (0, 4, 5, 6):
                u = pkg.electric_potential(pts[p], e, d["it"][k, r], d["gamma"][k], d["kappa"][k])
                assert abs(u - d["pot"][k, p, r]) <= TOL * abs(d["pot"][k, p, r])
                va = pkg.magnetic_potential(pts[p], e, d["il"][k, r], d["gamma"][k])
                assert _close(va, d["vecpot"][k, p, r]) <= TOL
                ve = pkg.electric_field(pts[p], e, d["il"][k, r], d["it"][k, r], d["gamma"][k], d["s"][k],
                                        d["kappa"][k], ve=[9.0, 9.0, 9.0])          # overwritten when |s| > 0
                assert _close(ve, d["efield"][k, p, r]) <= TOL
                ve0 = pkg.electric_field(pts[p], e, d["il"][k, r], d["it"][k, r], d["gamma"][k], 0.0, d["kappa"][k],
                                         ve=d["ve0"])                                 # added to when s = 0
                assert _close(ve0, d["efield_s0"][k, p, r]) <= TOL
            for l in range(d["paths"].shape[0]):
                v = pkg.voltage(d["paths"][l, :3], d["paths"][l, 3:], e, d["il"][k, r], d["it"][k, r], d["gamma"][k],
                                d["s"][k], d["kappa"][k])
                assert abs(v - d["voltage"][k, l, r]) <= 1e-8 * abs(d["voltage"][k, l, r])


def test_voltage_batch_matches_reference_fixture(gpu_pkg):
    pkg = gpu_pkg
    d = _field_case()
    v = pkg.voltage_batch(d["paths"], d["elec"], d["il"], d["it"], d["gamma"], d["s"], d["kappa"])
    assert v.shape == d["voltage"].shape
    assert _close(v, d["voltage"], axis=(1, 2)) <= 1e-8


def test_gpd_mhem_matches_oracle(gpu_pkg, port):
    pkg = gpu_pkg
    d = _field_case()
    rng = np.random.default_rng(3)
    pts = np.column_stack([rng.uniform(-6, 10, 40), rng.uniform(-6, 10, 40), np.zeros(40)])
    got = pkg.gpd_mhem_batch(pts, d["elec"], d["it"], d["gamma"], d["kappa"])
    for k in range(3):
        want = port.gpd_mhem(pts, d["elec"], d["it"][k].T, d["gamma"][k], d["kappa"][k])
        assert _close(got[k], want) <= 1e-12


def test_fields_many_samples_near_points_vs_oracle(gpu_pkg, port):
    """A sweep of 40 samples (60 Hz to 10 MHz, more than one warp of samples)
    at points from 1e-3 of an electrode length to far away, on a rod's axis
    beyond its tip and near a junction, against the oracle at 1e-12."""
    pkg = gpu_pkg
    from oracle import oracle as O
    grid, _ = pkg.electrode_grid(3, 3, 6.0, 6.0, 2, 2, 7e-3, -0.6)
    rod, _ = pkg.segment_electrode([6.0, 6.0, -0.6], [6.0, 6.0, -3.6], 2, 9e-3)
    e = np.vstack([grid, rod])
    m = e.shape[0]
    f = np.logspace(np.log10(60.0), 7, 40)
    s = 2j * np.pi * f + 1e3
    kappa = 1.0 / 150.0 + s * 9.0 * O.EPS0
    gamma = np.array([O.medium(a, b)[0] for a, b in zip(s, kappa)])
    rng = np.random.default_rng(21)
    il = rng.normal(size=(40, 1, m)) + 1j * rng.normal(size=(40, 1, m))
    it = rng.normal(size=(40, 1, m)) + 1j * rng.normal(size=(40, 1, m))
    pts = np.array([[1.5, 0.0015, -0.6], [1.5, 0.0, -0.603], [0.0, 0.0, -0.6 + 0.02], [6.0, 6.0, -3.7],
                    [6.0, 6.0, -5.0], [3.0, 2.9, -0.59], [2.0, 2.0, 0.0], [40.0, -30.0, 0.0]])
    out = pkg.fields_batch(pts, e, il, it, gamma, kappa)
    assert out["status"] == 0
    for k in (0, 13, 27, 39):
        for p in range(pts.shape[0]):
            u = port.electric_potential(pts[p], e, it[k, 0], gamma[k], kappa[k], 0, 1e-14, 1e-12)
            va = port.magnetic_potential(pts[p], e, il[k, 0], gamma[k], 1.0, 0, 1e-14, 1e-12)
            ve, _ = port.electric_field(pts[p], e, il[k, 0], it[k, 0], gamma[k], 0.0, kappa[k], 1.0, 0, 1e-14, 1e-12)
            assert abs(out["pot"][k, p, 0] - u) <= TOL * abs(u), (k, p)
            assert _close(out["vecpot"][k, p, 0], va) <= TOL, (k, p)
            assert _close(out["efield"][k, p, 0], ve) <= 1e-8, (k, p)


def test_point_on_electrode_is_flagged(gpu_pkg):
    pkg = gpu_pkg
    d = _field_case()
    e = d["elec"]
    on = e[0, 6:9].copy()                      # the midpoint of the first segment
    pkg.lib().tags_gpu_set_quiet(1)
    try:
        out = pkg.fields_batch(np.array([on, [9.0, 9.0, 0.0]]), e, d["il"], d["it"], d["gamma"], d["kappa"])
    finally:
        pkg.lib().tags_gpu_set_quiet(0)
    assert out["status"] == pkg.E_GEOMETRY
    assert np.all(np.isnan(out["pot"][:, 0]))
    assert np.all(np.isfinite(out["pot"][:, 1]))


def test_empty_and_zero_currents(gpu_pkg):
    pkg = gpu_pkg
    d = _field_case()
    z = np.zeros_like(d["il"])
    out = pkg.fields_batch(d["points"], d["elec"], z, z, d["gamma"], d["kappa"])
    assert not np.any(out["pot"]) and not np.any(out["vecpot"]) and not np.any(out["efield"])
    out = pkg.fields_batch(d["points"], d["elec"][:0], z[:, :, :0], z[:, :, :0], d["gamma"], d["kappa"])
    assert out["pot"].shape == (3, d["points"].shape[0], 2) and not np.any(out["pot"])


def test_more_injections_than_one_pass(gpu_pkg, port):
    """Six injections (the kernel takes four per pass over the electrodes) and
    a single sample: every injection against the oracle."""
    pkg = gpu_pkg
    d = _field_case()
    rng = np.random.default_rng(8)
    m = d["elec"].shape[0]
    il = rng.normal(size=(1, 6, m)) + 1j * rng.normal(size=(1, 6, m))
    it = rng.normal(size=(1, 6, m)) + 1j * rng.normal(size=(1, 6, m))
    pts = d["points"][:4]
    out = pkg.fields_batch(pts, d["elec"], il, it, d["gamma"][1:2], d["kappa"][1:2])
    for r in range(6):
        for p in range(pts.shape[0]):
            u = port.electric_potential(pts[p], d["elec"], it[0, r], d["gamma"][1], d["kappa"][1], 0, 1e-14, 1e-12)
            va = port.magnetic_potential(pts[p], d["elec"], il[0, r], d["gamma"][1], 1.0, 0, 1e-14, 1e-12)
            assert abs(out["pot"][0, p, r] - u) <= TOL * abs(u)
            assert _close(out["vecpot"][0, p, r], va) <= TOL


@pytest.mark.parametrize("x", [0.05, 0.3, 0.6, 1.9, 2.1, 5.0])
@pytest.mark.parametrize("ns,nrhs,m,P", [(1, 1, 1, 3), (3, 5, 7, 4), (33, 2, 40, 2), (130, 1, 3, 1)])
def test_field_series_and_its_limits_match_oracle(gpu_pkg, port, x, ns, nrhs, m, P):
    """Moment series with 12, 16 and 24 terms and the rule per sample past
    their reach (x = |gamma| (L + L/8) / 2, 2.0), mixed in one call: the last
    sample is ten times higher. Points near (within 2 L of) and far from the
    electrodes; oracle at 1e-11, TOL of the largest magnitude."""
    pkg = gpu_pkg
    rng = np.random.default_rng(m)
    e, _ = pkg.segment_electrode([0.0, 0.0, -0.5], [1.0 * m, 0.0, -0.5], m, 7e-3)
    pts = np.stack([np.linspace(-0.3, 1.1 * m, P), np.full(P, 0.2), np.linspace(0.0, 30.0, P) - 0.4], axis=1)
    gamma = x / 0.5625 * np.exp(0.25j * np.pi) * np.linspace(0.5, 1.0, ns)
    if ns > 1:
        gamma[-1] *= 10
    kappa = np.full(ns, 0.01 + 1e-3j)
    il, it = (rng.standard_normal((ns, nrhs, m)) + 1j * rng.standard_normal((ns, nrhs, m)) for _ in range(2))
    il[0, 0, 0] = 1e-17                     # below DBL_EPSILON: skipped in the vector potential and the field
    it[0, 0, 0] = 1e-17
    out = pkg.fields_batch(pts, e, il, it, gamma, kappa)
    assert out["status"] == 0
    for k in sorted({0, ns // 2, ns - 1}):
        for r in range(nrhs):
            for p in range(P):
                u = port.electric_potential(pts[p], e, it[k, r], gamma[k], kappa[k], req_abs=0.0, req_rel=1e-11)
                va = port.magnetic_potential(pts[p], e, il[k, r], gamma[k], req_abs=0.0, req_rel=1e-11)
                ve, _ = port.electric_field(pts[p], e, il[k, r], it[k, r], gamma[k], 0.0, kappa[k], req_abs=0.0,
                                            req_rel=1e-11)
                # e^{-gamma r} underflows at the far points of the high samples: what is below the
                # smallest normal number carries fewer than 53 bits on either side
                for got, want in ((out["pot"][k, p, r], u), (out["vecpot"][k, p, r], va), (out["efield"][k, p, r], ve)):
                    assert np.max(np.abs(got - want)) <= TOL * np.max(np.abs(want)) + np.finfo(float).tiny


@pytest.mark.parametrize("m,P,ns", [(1, 1, 1), (5, 1, 2), (63, 1, 1), (64, 1, 3), (130, 2, 40)])
def test_field_of_few_points_and_many_electrodes_matches_oracle(gpu_pkg, port, m, P, ns):
    """Lanes per pair from 32 down to 1, chunks summed by a thread or a warp; oracle at 1e-11, TOL of the largest
    magnitude."""
    test_field_series_and_its_limits_match_oracle(gpu_pkg, port, 0.05, ns, 2, m, P)


def fine_rule(point, e, gamma):
    """The integrals of e^{-gamma r}/r and of (1 + gamma r) e^{-gamma r} / r^3 (point - position) over an electrode,
    panels halving towards the point, 32 nodes each."""
    a, b = e[:3], e[3:6]
    x, w = np.polynomial.legendre.leggauss(32)
    foot = np.clip((point - a) @ (b - a) / ((b - a) @ (b - a)), 0.0, 1.0)
    edges = np.unique(np.clip(np.concatenate([[0.0, 1.0, foot], foot + 2.0 ** -np.arange(12), foot - 2.0 ** -np.arange(12)]),
                              0.0, 1.0))
    j, f = 0.0, np.zeros(3, np.complex128)
    for lo, hi in zip(edges[:-1], edges[1:]):
        t = lo + (hi - lo) * (x + 1) / 2
        d = point - (a + t[:, None] * (b - a))
        r = np.linalg.norm(d, axis=1)
        ex = w * (hi - lo) / 2 * np.exp(-gamma * r)
        j = j + (ex / r).sum()
        f = f + ((ex * (1 + gamma * r) / r ** 3)[:, None] * d).sum(axis=0)
    return j, f


@pytest.mark.parametrize("x", [0.05, 0.36, 0.54, 0.6, 0.99, 1.1, 1.5, 1.99])
@pytest.mark.parametrize("m", [1, 5, 70])
def test_field_series_to_rounding_at_every_order(gpu_pkg, x, m):
    """Points along the axis and abeam on both sides of every distance at which the series' rule changes its order, x =
    |gamma| (L + L/8) / 2 up to the reach of 2: 1e-14 of the value (some ten roundings of the 24 terms' sum, whose
    largest is e^2 times the first) and the rounding of the phase |gamma| r on either side. One electrode carries the
    current, so that no two cancel."""
    pkg = gpu_pkg
    e, _ = pkg.segment_electrode([0.0, 0.0, -0.5], [1.0 * m, 0.0, -0.5], m, 7e-3)
    gamma = x / 0.5625 * np.exp(0.25j * np.pi)
    k = m // 2
    mid = np.array([k + 0.5, 0.0, -0.5])
    pts = []
    for dist in (0.4, 1.9, 2.1, 3.9, 4.1, 7.9, 8.1, 15.9, 16.1, 20.0):
        for turn in (0.0, 0.6, np.pi / 2):
            step = np.array([np.cos(turn), np.sin(turn), 0.0])
            pts.append(mid + (dist + 0.5 * abs(step[0])) * step + np.array([0.0, 1e-3 if turn == 0.0 else 0.0, 0.0]))
    pts = np.array(pts)
    if m > 1:
        pts[:, 2] += 0.03                   # off the axis of the other electrodes
    cur = np.zeros((1, 1, m), np.complex128)
    cur[0, 0, k] = 1.0
    out = pkg.fields_batch(pts, e, cur, cur, [gamma], [1.0 + 0j])
    assert out["status"] == 0
    for p, point in enumerate(pts):
        j, f = fine_rule(point, e[k], gamma)
        tol = 1e-14 + 2 * np.finfo(float).eps * abs(gamma) * (np.linalg.norm(point - mid) + 0.5)
        assert abs(4 * np.pi * out["pot"][0, p, 0] - j) <= tol * abs(j)
        assert np.abs(4 * np.pi * out["efield"][0, p, 0] - f).max() <= tol * np.abs(f).max()


@pytest.mark.parametrize("dist,P,m", [(1000.0, 1, 10), (1000.0, 3, 1), (300.0, 40, 8), (30.0, 70, 4)])
@pytest.mark.parametrize("ns", [1, 40, 130])
def test_field_far_away_matches_fine_rule(gpu_pkg, dist, P, m, ns):
    """Few pairs far apart, where most of the expansion centres between them are not used, and more pairs than centres:
    exponentials formed per pair and from the table. Tolerance as in the test above, for m currents of one sign."""
    pkg = gpu_pkg
    e, _ = pkg.segment_electrode([0.0, 0.0, -0.5], [1.0 * m, 0.0, -0.5], m, 7e-3)
    gamma = 0.02 * np.exp(0.25j * np.pi) * np.linspace(0.1, 1.0, ns)
    pts = np.stack([np.linspace(dist, dist + 2.0, P), np.full(P, 0.3), np.zeros(P)], axis=1)
    cur = np.ones((ns, 1, m), np.complex128)
    out = pkg.fields_batch(pts, e, cur, cur, gamma, np.ones(ns, np.complex128))
    assert out["status"] == 0
    for k in {0, ns // 2, ns - 1}:
        for p in {0, P - 1}:
            j, f = (sum(v) for v in zip(*(fine_rule(pts[p], e[q], gamma[k]) for q in range(m))))
            tol = 1e-14 + 2 * np.finfo(float).eps * abs(gamma[k]) * (dist + 2 + m)
            assert abs(4 * np.pi * out["pot"][k, p, 0] - j) <= tol * abs(j)
            assert np.abs(4 * np.pi * out["efield"][k, p, 0] - f).max() <= tol * np.abs(f).max()


def test_field_memory_follows_the_work(gpu_pkg):
    """A call of many samples and few pairs takes device memory for its samples, inputs and outputs, some 1 KB a sample
    here, not for a table of every distance in between (64 KB a sample)."""
    torch = pytest.importorskip("torch")
    pkg = gpu_pkg
    m, ns = 2, 200000
    e, _ = pkg.segment_electrode([0.0, 0.0, -0.5], [1.0 * m, 0.0, -0.5], m, 7e-3)
    cur = np.ones((ns, 1, m), np.complex128)
    before = torch.cuda.mem_get_info()[0]
    out = pkg.fields_batch([[1000.0, 0.0, 0.0]], e, cur, cur, np.full(ns, 0.01 + 0.01j), np.ones(ns, np.complex128))
    assert out["status"] == 0 and np.ptp(out["pot"].real) == 0.0
    assert before - torch.cuda.mem_get_info()[0] < 1 << 30


def check_against_fine_rule(out, pts, e, il, it, gamma, samples, points):
    """Potential, vector potential and field of the given samples and points to 1e-12 of the summed magnitudes."""
    for k in samples:
        for p in points:
            pairs = [fine_rule(pts[p], seg, gamma[k]) for seg in e]
            j = np.array([v[0] for v in pairs])
            f = np.array([v[1] for v in pairs])
            d = e[:, 3:6] - e[:, :3]
            for r in range(il.shape[1]):
                for got, want, size in (
                        (4 * np.pi * out["pot"][k, p, r], it[k, r] @ j, np.abs(it[k, r]) @ np.abs(j)),
                        (1e7 * out["vecpot"][k, p, r], (il[k, r] * j) @ d, np.abs(il[k, r] * j) @ np.abs(d).max(axis=1)),
                        (4 * np.pi * out["efield"][k, p, r], it[k, r] @ f, np.abs(it[k, r]) @ np.abs(f).max(axis=1))):
                    assert np.max(np.abs(got - want)) <= 1e-12 * size


@pytest.mark.parametrize("ns,far", [(80, (40,)), (96, (3, 95)), (70, (66,)), (200, (130, 131))])
def test_field_call_with_both_kernels_matches_fine_rule(gpu_pkg, ns, far):
    """Some groups of 32 samples hold one past the series' reach and take the rule per sample, the others the series, in
    one call with a partial last group and five injections. The evaluations counted are those of calls of the former
    groups alone, so both kernels had their part."""
    pkg = gpu_pkg
    rng = np.random.default_rng(ns)
    m, P, R = 40, 36, 5
    e, _ = pkg.segment_electrode([0.0, 0.0, -0.5], [1.0 * m, 0.0, -0.5], m, 7e-3)
    pts = np.stack([np.linspace(-0.3, 50.0, P), np.full(P, 0.2), np.linspace(0.0, 3.0, P) - 0.4], axis=1)
    gamma = 0.9 / 0.5625 * np.exp(0.25j * np.pi) * np.linspace(0.2, 1.0, ns)
    gamma[list(far)] *= 10 / np.abs(gamma[list(far)])
    il, it = (rng.standard_normal((ns, R, m)) + 1j * rng.standard_normal((ns, R, m)) for _ in range(2))
    kappa = np.ones(ns, np.complex128)
    pkg.fields_evaluations(reset=True)
    out = pkg.fields_batch(pts, e, il, it, gamma, kappa)
    together = pkg.fields_evaluations(reset=True)
    assert out["status"] == 0
    rule = sorted({f // 32 for f in far})
    for g in rule:
        take = slice(32 * g, min(ns, 32 * g + 32))
        # alone, a last group of fewer is shared out differently (G samples per warp), but evaluates the same nodes
        alone = pkg.fields_batch(pts, e, il[take], it[take], gamma[take], kappa[take])
        assert rel(alone["efield"], out["efield"][take]) < 1e-12
    assert 0 < pkg.fields_evaluations(reset=True) == together
    check_against_fine_rule(out, pts, e, il, it, gamma, sorted({0, ns - 1, far[0], far[0] - 1, 32 * (far[0] // 32) - 1}),
                            (0, P - 1))


def rel(a, b):
    return float(np.max(np.abs(a - b)) / np.max(np.abs(b)))


@pytest.mark.parametrize("x", [0.04, 0.085, 0.1, 0.3, 0.36, 0.38, 1.2])
@pytest.mark.parametrize("ns,m", [(5, 3), (40, 33)])
def test_field_series_of_many_samples_at_every_term_count(gpu_pkg, x, ns, m):
    """Calls of several samples whose largest needs up to 12, 16 and 24 terms (x = 0.09 and 0.37 part them)."""
    pkg = gpu_pkg
    rng = np.random.default_rng(m)
    e, _ = pkg.segment_electrode([0.0, 0.0, -0.5], [1.0 * m, 0.0, -0.5], m, 7e-3)
    pts = np.stack([np.linspace(-0.3, 1.4 * m, 6), np.full(6, 0.2), np.linspace(0.0, 3.0, 6) - 0.4], axis=1)
    gamma = x / 0.5625 * np.exp(0.25j * np.pi) * np.linspace(0.2, 1.0, ns)
    il, it = (rng.standard_normal((ns, 5, m)) + 1j * rng.standard_normal((ns, 5, m)) for _ in range(2))
    pkg.fields_evaluations(reset=True)
    out = pkg.fields_batch(pts, e, il, it, gamma, np.ones(ns, np.complex128))
    assert out["status"] == 0 and pkg.fields_evaluations() == 0
    check_against_fine_rule(out, pts, e, il, it, gamma, {0, ns // 2, ns - 1}, (0, 2, 5))
