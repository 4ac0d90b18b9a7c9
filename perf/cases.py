"""The measured cases: what a user of this library has it do, through its public
entry points, from one rod's harmonic impedance to a 17875-unknown grid.

Every case is a dict of plain values; its "kind" names the work:

plan        Plan.run: solutions [U; I_L; I_T] of a grid or rod for Laplace samples
dropin      the reference's per-sample chain on host arrays: calculate_impedances,
            impedances_images, fill_impedance_imm, solve_immittance
admittance  the examples' nodal chain on host arrays: calculate_yla_ytb,
            fill_impedance_adm2, solve_admittance
grids       GridBatch.run: many grids of uneven size, many samples, one call
fields      fields_batch: potential, vector potential and field on a line of points
voltage     voltage_batch: step and touch voltages along straight paths
inlt        inv_laplace_batch: transients of many nodes from their spectra
"""
import importlib
import math

import numpy as np
import torch

tags = importlib.import_module("transient-analysis-grounding-systems_gb300")

NT_BAND = 4094              # the 2048-sample transient job: nt, window (s)
T_BAND = 2047 / 1e7


# ---- the cases ---------------------------------------------------------------------

def listed():
    return [
        # harmonic impedance of one vertical rod over 100 frequencies: the smallest system
        {"name": "rod_plain_100f", "kind": "plan", "shape": "rod", "segments": 10, "precision": "plain",
         "ns": 100, "batch": 100, "soil": "constant", "band": "log"},
        # one frequency of a 100-segment grid by a C caller's relinked loop body
        {"name": "grid100_dropin", "kind": "dropin", "shape": "grid", "meshes": 4, "nx": 2, "ny": 3, "side": 10.0},
        # one frequency of the mHEM examples' loop body, 10 x 10 meshes
        {"name": "grid220_admittance", "kind": "admittance", "shape": "grid", "meshes": 10, "nx": 1, "ny": 1,
         "side": 20.0},
        # transient of the 100-segment grid in full FP64
        {"name": "grid100_plain", "kind": "plan", "shape": "grid", "meshes": 4, "nx": 2, "ny": 3, "side": 10.0,
         "precision": "plain", "ns": 256, "batch": 256, "soil": "constant", "band": "laplace"},
        # transient of the 100-segment grid, mixed precision, all 1024 samples
        {"name": "grid100_mixed", "kind": "plan", "shape": "grid", "meshes": 4, "nx": 2, "ny": 3, "side": 10.0,
         "precision": "mixed", "ns": 1024, "batch": 256, "soil": "constant", "band": "laplace"},
        # the 60 x 60 m grid, every 16th of its 2048 samples, frequency-dependent soil
        {"name": "grid1560_mixed", "kind": "plan", "shape": "grid", "meshes": 12, "nx": 5, "ny": 5, "side": 60.0,
         "precision": "mixed", "ns": 128, "batch": 128, "soil": "alipio", "band": "laplace"},
        # the same grid in full FP64: the accuracy check of the mixed form
        {"name": "grid1560_plain", "kind": "plan", "shape": "grid", "meshes": 12, "nx": 5, "ny": 5, "side": 60.0,
         "precision": "plain", "ns": 2, "batch": 2, "soil": "alipio", "band": "laplace"},
        # a design study: many candidate grids of uneven size at once
        {"name": "uneven_grids", "kind": "grids", "count": 16, "draw": 7, "ns": 64},
        # a substation-size grid with rods, eight samples resident
        {"name": "rods17875_mixed", "kind": "plan", "shape": "rods", "vertices": 25, "side": 120.0, "nx": 5,
         "rods": 50, "rod_segments": 3, "precision": "mixed", "ns": 8, "batch": 8, "soil": "alipio",
         "band": "laplace"},
        # ground-level field profile over the 60 x 60 m grid, four injections
        {"name": "field_line_1560", "kind": "fields", "shape": "grid", "meshes": 12, "nx": 5, "ny": 5, "side": 60.0,
         "points": 251, "nrhs": 4, "ns": 64},
        # step and touch voltages of the 100-segment grid
        {"name": "voltages_grid100", "kind": "voltage", "shape": "grid", "meshes": 4, "nx": 2, "ny": 3, "side": 10.0,
         "paths": 40, "nrhs": 1, "ns": 128},
        # transients of all nodes of the 60 x 60 m grid
        {"name": "inlt_1417_nodes", "kind": "inlt", "nt": NT_BAND, "series": 1417, "filter": 0},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _segments(c):
    return c["meshes"] * (c["meshes"] + 1) * (c["nx"] + c["ny"])


def _draw_grid(rng, most):
    """A grid of 4 .. most segments, sides 5-60 m as the uneven workload's and the large grid's."""
    target = _log_int(rng, 4, most)
    while True:
        c = {"shape": "grid", "meshes": rng.randint(1, 12), "nx": rng.randint(1, 5), "ny": rng.randint(1, 5),
             "side": round(rng.uniform(5.0, 60.0), 2)}
        m = _segments(c)
        edge = c["side"] / c["meshes"]
        if target / 2 <= m <= target * 1.5 + 2 and m <= most and 0.4 <= edge / max(c["nx"], c["ny"]) and \
                edge / min(c["nx"], c["ny"]) <= 12.0:
            return c


def draw(rng):
    kind = rng.choice(["plan", "plan", "plan", "dropin", "admittance", "grids", "fields", "voltage", "inlt"])
    if kind == "plan":
        size = rng.choice(["rod", "small", "small", "large", "rods"])
        if size == "rod":
            ns = _log_int(rng, 1, 400)
            return {"kind": kind, "shape": "rod", "segments": _log_int(rng, 1, 60),
                    "precision": rng.choice(["plain", "mixed"]), "ns": ns, "batch": max(1, ns // rng.randint(1, 3)),
                    "soil": rng.choice(["constant", "alipio"]), "band": "log"}
        if size == "rods":
            return {"kind": kind, "shape": "rods", "vertices": rng.randint(4, 16), "side": 80.0, "nx": rng.randint(3, 5),
                    "rods": rng.randint(2, 12), "rod_segments": rng.randint(1, 3), "precision": "mixed",
                    "ns": rng.randint(1, 8), "batch": 8, "soil": "alipio", "band": "laplace"}
        c = _draw_grid(rng, 400 if size == "small" else 1560)
        m = _segments(c)
        plain = rng.random() < 0.4
        # no more work than the listed cases of the same precision
        most = max(1, min(512, int((2 if plain else 128) * (1560 / m) ** 2.5)))
        ns = _log_int(rng, 1, most)
        return {"kind": kind, **c, "precision": "plain" if plain else "mixed", "ns": ns,
                "batch": max(1, ns // rng.randint(1, 3)),
                "soil": rng.choice(["constant", "alipio"]) if m <= 900 else "alipio", "band": "laplace"}
    if kind == "dropin":
        return {"kind": kind, **_draw_grid(rng, 400)}
    if kind == "admittance":
        return {"kind": kind, **_draw_grid(rng, 400)}
    if kind == "grids":
        return {"kind": kind, "count": rng.randint(2, 16), "draw": rng.randint(0, 1000), "ns": _log_int(rng, 4, 64)}
    if kind == "fields":
        return {"kind": kind, **_draw_grid(rng, 1560), "points": _log_int(rng, 1, 251), "nrhs": rng.randint(1, 4),
                "ns": _log_int(rng, 1, 64)}
    if kind == "voltage":
        return {"kind": kind, **_draw_grid(rng, 400), "paths": _log_int(rng, 1, 60), "nrhs": rng.randint(1, 3),
                "ns": _log_int(rng, 1, 128)}
    return {"kind": "inlt", "nt": _log_int(rng, 5, 4096), "series": _log_int(rng, 1, 1417),
            "filter": rng.choice([0, 0, 1, 2, 4])}


# ---- inputs ------------------------------------------------------------------------

def _geometry(case):
    """Electrodes, images, nodes and the injection node."""
    if case["shape"] == "rod":
        elec, nodes = tags.segment_electrode([0.0, 0.0, 0.0], [0.0, 0.0, -0.3 * case["segments"]], case["segments"],
                                             7e-3)
        return elec, tags.images(elec), nodes, 0
    if case["shape"] == "rods":
        elec, nodes = tags.grid_with_rods(vertices=case["vertices"], length=case["side"], edge_segments=case["nx"],
                                          rods=case["rods"], rod_segments=case["rod_segments"])
    else:
        v, a = case["meshes"] + 1, case["side"]
        elec, nodes = tags.electrode_grid(v, v, a, a, case["nx"], case["ny"], 7e-3, -0.5)
    inj = int(np.argmin(np.linalg.norm(nodes - [case["side"] / 2, case["side"] / 2, -0.5], axis=1)))
    return elec, tags.images(elec), nodes, inj


def _kappa(s, soil, rng):
    """kappa(s) of a soil: constant, of 50-5000 ohm m, or the Alipio-Visacro frequency dependence over 100-1000 ohm m."""
    lo, hi = (50.0, 5000.0) if soil == "constant" else (100.0, 1000.0)
    sigma0 = 1.0 / math.exp(rng.uniform(math.log(lo), math.log(hi)))
    if soil == "constant":
        return sigma0 + s * tags.EPS0 * rng.uniform(5.0, 40.0)
    h, g, f = 1.26 * (sigma0 * 1e3) ** -0.73, 0.54, s / (2j * math.pi)
    t = math.tan(math.pi * g / 2) / (2 * math.pi * tags.EPS0 * 1e6 ** g)
    return sigma0 + sigma0 * h * (f / 1e6) ** g + s * tags.EPS0 * (12.0 + t * sigma0 * h * f ** (g - 1.0))


def _samples(case, rng):
    """s, kappa (ns,): log-spaced frequencies 100 Hz - 10 MHz, or Laplace samples strided over the band to 10 MHz."""
    ns = case["ns"]
    if case["band"] == "log":
        s = 2j * math.pi * np.logspace(2, 7, ns) * rng.uniform(0.9, 1.0)
    else:
        k = (np.arange(ns) * 2048) // ns
        s = math.log(float(NT_BAND) ** 2) / T_BAND + 2j * math.pi / T_BAND * k
    return s, _kappa(s, case["soil"], rng)


def _inputs(case, seed):
    """The host arrays of a case: all that its result depends on."""
    rng = np.random.default_rng([seed, 2021])
    kind, d = case["kind"], {}
    if kind == "inlt":
        nt, nser = case["nt"], case["series"]
        tmax = (nt // 2) / 1e7
        s = math.log(float(nt) ** 2) / tmax + 2j * math.pi / tmax * np.arange(nt // 2 + 1)
        # double-exponential injections through first-order impedances
        a, b = rng.uniform(1e4, 5e4, nser), rng.uniform(1e6, 5e6, nser)
        tau, r = rng.uniform(1e-7, 1e-6, nser), rng.uniform(1.0, 50.0, nser)
        g = (r * 1e3) * (1 / (s[:, None] + a) - 1 / (s[:, None] + b)) / (1 + s[:, None] * tau)
        return {"nt": nt, "tmax": tmax, "s": s, "g": np.ascontiguousarray(g), "filter": case["filter"]}
    if kind == "grids":
        jobs = []
        for g in tags.uneven_grids(case["count"], case["draw"]):
            s = math.log(float(NT_BAND) ** 2) / T_BAND + 2j * math.pi / T_BAND * ((np.arange(case["ns"]) * 2048) //
                                                                                   case["ns"])
            jobs.append({"electrodes": g["electrodes"], "images": tags.images(g["electrodes"]), "nodes": g["nodes"],
                         "s": s, "kappa": _kappa(s, "constant", rng), "inj_node": 0})
        return {"jobs": jobs}
    d["elec"], d["img"], d["nodes"], d["inj"] = _geometry(case)
    m, n = len(d["elec"]), len(d["nodes"])
    if kind == "plan":
        d["s"], d["kappa"] = _samples(case, rng)
        return d
    if kind in ("dropin", "admittance"):
        s = np.array([rng.uniform(1e4, 1e5) + 2j * math.pi * math.exp(rng.uniform(math.log(1e3), math.log(1e7)))])
        d["s"], d["kappa"] = s, _kappa(s, "constant", rng)
        return d
    # segment currents as a solve returns them: complex, 1/m of the injected ampere and up
    k = (np.arange(case["ns"]) * 2048) // case["ns"]
    d["s"] = math.log(float(NT_BAND) ** 2) / T_BAND + 2j * math.pi / T_BAND * k
    d["kappa"] = _kappa(d["s"], "constant", rng)
    d["gamma"] = np.sqrt(d["s"] * tags.MU0 * d["kappa"])
    shape = (case["ns"], case["nrhs"], m)
    for name in ("il", "it"):
        d[name] = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)) / m
    side = case["side"]
    if kind == "fields":
        x = np.linspace(-0.2 * side, 1.2 * side, case["points"]) if case["points"] > 1 else np.array([0.37 * side])
        d["points"] = np.stack([x, 0.43 * side + 0.1 * x, np.zeros_like(x)], axis=1)
    else:
        p = np.concatenate([rng.uniform(-0.1 * side, 1.1 * side, (case["paths"], 2)), np.zeros((case["paths"], 1))], 1)
        ang = rng.uniform(0, 2 * math.pi, case["paths"])
        d["paths"] = np.concatenate([p, p + np.stack([np.cos(ang), np.sin(ang), 0 * ang], 1)], 1)   # 1 m steps
    return d


def _mhem_potentials(d):
    """zl, zt of the mHEM model at one sample (column-major, lower triangle), as the examples rescale them."""
    elec, img, m = d["elec"], d["img"], len(d["elec"])
    gamma, ref_t = tags.medium(d["s"][0], d["kappa"][0])
    pots = [np.zeros(m * m, np.complex128) for _ in range(4)]
    tags.calculate_impedances(pots[0], pots[1], elec, 0, 0, 0, 0, integration_type=tags.INTG_MHEM)
    tags.impedances_images(pots[2], pots[3], elec, img, 0, 0, 0, 0, 0, 0, integration_type=tags.INTG_MHEM)
    mid, mim = elec[:, 6:9], img[:, 6:9]
    direct = np.exp(-gamma * np.linalg.norm(mid[:, None] - mid[None], axis=2)).ravel()
    image = np.exp(-gamma * np.linalg.norm(mim[:, None] - mid[None], axis=2)).ravel()
    zl = (direct * pots[0] + image * pots[2]) * (d["s"][0] * tags.MU0 / tags.FOUR_PI)
    zt = (direct * pots[1] + ref_t * image * pots[3]) / (tags.FOUR_PI * d["kappa"][0])
    return zl, zt


def prepare(case, seed):
    d = _inputs(case, seed)
    kind = case["kind"]
    d["kind"] = kind
    if kind == "plan":
        prec = tags.PLAIN_FP64 if case["precision"] == "plain" else tags.MIXED
        d["plan"] = tags.Plan(d["elec"], d["img"], d["nodes"], prec, case["batch"])
    elif kind == "grids":
        d["batch"] = tags.GridBatch(d["jobs"], tags.MIXED, max_batch=case["ns"])
    elif kind == "dropin":
        m, n = len(d["elec"]), len(d["nodes"])
        d["gamma"], d["ref_t"] = tags.medium(d["s"][0], d["kappa"][0])
        d["zl"], d["zt"] = np.zeros(m * m, np.complex128), np.zeros(m * m, np.complex128)
        d["wg"] = np.zeros((n + 2 * m) ** 2, np.complex128)
        tags.fill_incidence_imm(d["wg"], d["elec"], d["nodes"])      # once per geometry
    elif kind == "admittance":
        m, n = len(d["elec"]), len(d["nodes"])
        d["zl0"], d["zt0"] = _mhem_potentials(d)
        for name, size in (("a", m * n), ("b", m * n), ("yla", m * n), ("ytb", m * n), ("yn", n * n), ("zl", m * m),
                           ("zt", m * m)):
            d[name] = np.zeros(size, np.complex128)
        tags.fill_incidence_adm(d["a"], d["b"], d["elec"], d["nodes"])
    return d


def run(d):
    kind = d["kind"]
    if kind == "plan":
        sol, info, _ = d["plan"].run(d["s"], d["kappa"], inj_node=d["inj"])
        return {"sol": sol, "info": info}
    if kind == "grids":
        out, _ = d["batch"].run(d["jobs"])
        return [{"sol": sol, "info": info} for sol, info in out]
    if kind == "dropin":
        m, n, s, k = len(d["elec"]), len(d["nodes"]), d["s"][0], d["kappa"][0]
        x = np.zeros(n + 2 * m, np.complex128)
        x[d["inj"]] = 1.0
        rc = [tags.calculate_impedances(d["zl"], d["zt"], d["elec"], d["gamma"], s, 1.0, k),
              tags.impedances_images(d["zl"], d["zt"], d["elec"], d["img"], d["gamma"], s, 1.0, k, 1.0, d["ref_t"]),
              tags.fill_impedance_imm(d["wg"], d["zl"], d["zt"], m, n),
              tags.solve_immittance(d["wg"], x, m, n)]
        return {"zl": d["zl"], "zt": d["zt"], "x": x, "rc": np.array(rc)}
    if kind == "admittance":
        m, n = len(d["elec"]), len(d["nodes"])
        np.copyto(d["zl"], d["zl0"])                                 # the call leaves the inverses there
        np.copyto(d["zt"], d["zt0"])
        x = np.zeros(n, np.complex128)
        x[d["inj"]] = 1.0
        rc = [tags.calculate_yla_ytb(d["yla"], d["ytb"], d["zl"], d["zt"], d["a"], d["b"], m, n),
              tags.fill_impedance_adm2(d["yn"], d["yla"], d["ytb"], d["a"], d["b"], m, n),
              tags.solve_admittance(d["yn"], x, n)]
        return {"yla": d["yla"], "ytb": d["ytb"], "yn": d["yn"], "x": x, "rc": np.array(rc)}
    if kind == "fields":
        return tags.fields_batch(d["points"], d["elec"], d["il"], d["it"], d["gamma"], d["kappa"])
    if kind == "voltage":
        return tags.voltage_batch(d["paths"], d["elec"], d["il"], d["it"], d["gamma"], d["s"], d["kappa"])
    return tags.inv_laplace_batch(d["g"], d["s"], d["tmax"], d["nt"], d["filter"])


# ---- what a pass cannot do without -------------------------------------------------

PAIR_FLOPS = 100.0           # one pair integral of e^{-gamma r}/r and its two entries
NODE_FLOPS = 60.0            # one point-electrode integral of the potential and the field


def _solve_work(m, n, ns):
    """Direct and image integrals of the lower triangle, and the symmetric elimination of
    [-ZL, -ZT] into the node block (their coupling block is zero), in real flops."""
    fill = m * m * PAIR_FLOPS
    elim = 2 * (4 / 3 * m ** 3 + 4 * m * m * n + 4 * m * n * n) + 4 / 3 * n ** 3
    return {"bytes": ns * (16 * (n + 2 * m) + 32) + 176 * m + 24 * n, "flops": ns * (fill + elim)}


def _sizes(case):
    if case["shape"] == "rod":
        return case["segments"], case["segments"] + 1
    if case["shape"] == "rods":
        v, e = case["vertices"], case["nx"]
        return 2 * e * v * (v - 1) + case["rods"] * case["rod_segments"], \
            v * v + 2 * v * (v - 1) * (e - 1) + case["rods"] * case["rod_segments"]
    v = case["meshes"] + 1
    return _segments(case), tags.number_nodes(v, v, case["nx"], case["ny"])


def work(case):
    kind = case["kind"]
    if kind == "plan":
        return _solve_work(*_sizes(case), case["ns"])
    if kind == "grids":
        parts = [_solve_work(len(g["electrodes"]), len(g["nodes"]), case["ns"])
                 for g in tags.uneven_grids(case["count"], case["draw"])]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind == "inlt":
        nt, nser = case["nt"], case["series"]
        return {"bytes": nser * (16 * (nt // 2 + 1) + 8 * nt), "flops": 2.5 * nser * nt * math.log2(nt)}
    m, n = _sizes(case)
    if kind == "dropin":
        w = _solve_work(m, n, 1)
        return {"bytes": 2 * 16 * m * m + 16 * (n + 2 * m) ** 2 + 16 * (n + 2 * m), "flops": w["flops"]}
    if kind == "admittance":
        return {"bytes": 4 * 16 * m * m + 4 * 16 * m * n + 16 * n * n + 16 * n, "flops": _solve_work(m, n, 1)["flops"]}
    ns, nrhs = case["ns"], case["nrhs"]
    if kind == "fields":
        p = case["points"]
        return {"bytes": 16 * ns * nrhs * (2 * m + 7 * p), "flops": ns * p * m * (NODE_FLOPS + 56 * nrhs)}
    p = case["paths"]
    return {"bytes": 16 * ns * nrhs * (2 * m + p), "flops": ns * p * m * (2 * NODE_FLOPS + PAIR_FLOPS + 24 * nrhs)}


# ---- 64-bit values, by plain quadrature and plain solves -----------------------------

DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(x):
    return torch.as_tensor(np.ascontiguousarray(x), device=DEV)


def _gauss(panels, order):
    x, w = np.polynomial.legendre.leggauss(order)
    x = (np.arange(panels)[:, None] + 0.5 * (x + 1)).ravel() / panels
    return _t(x), _t(np.tile(0.5 * w / panels, panels))


def _phi(x):
    """(1 - e^{-x}) / x, by its series where |x| is small."""
    small = x.abs() < 0.5
    y = torch.where(small, x, torch.zeros_like(x))
    acc = torch.ones_like(x)
    for k in range(18, 1, -1):
        acc = 1 - y * acc / k
    z = torch.where(small, torch.ones_like(x), x)
    return torch.where(small, acc, (1 - torch.exp(-z)) / z)


def _pair_integrals(recv, send, gamma):
    """Double line integrals of e^{-gamma r}/r over the unit squares of the pairs (recv[i], send[i]), (pairs, samples)."""
    ra, rb, sa, sb = _t(recv[:, :3]), _t(recv[:, 3:6]), _t(send[:, :3]), _t(send[:, 3:6])
    lr, ls = _t(recv[:, 9]), _t(send[:, 9])
    g = _t(np.atleast_1d(gamma))
    out = torch.zeros((len(recv), len(g)), dtype=torch.complex128, device=DEV)
    dist = ((ra + rb) / 2 - (sa + sb) / 2).norm(dim=1)
    touch = torch.zeros(len(recv), dtype=torch.bool, device=DEV)
    for p, q in ((ra, rb), (rb, ra)):                 # p: the receiver's shared end
        for u, v in ((sa, sb), (sb, sa)):
            hit = ((p - u).abs().amax(dim=1) < 1e-9) & ~touch
            touch |= hit
            ids = hit.nonzero()[:, 0]
            if not len(ids):
                continue
            x, w = _gauss(4, 24)
            d0, d1 = (q - p)[ids], (v - u)[ids]
            for e0, e1 in ((d0, d1), (d1, d0)):
                rho = (e0[:, None] - x[:, None] * e1[:, None]).norm(dim=2)
                for k in range(len(g)):
                    out[ids, k] += (w * _phi(g[k] * rho) / rho).sum(dim=1)
    far = dist > 5 * torch.maximum(lr, ls)
    longest = float(max(recv[:, 9].max(), send[:, 9].max()))
    reach = float(np.abs(gamma).max()) * longest
    near = (~far & ~touch).nonzero()[:, 0]
    closest = longest
    if len(near):
        q = torch.linspace(0, 1, 9, dtype=torch.float64, device=DEV)[None, :, None]
        pr = (ra[near, None] + q * (rb - ra)[near, None])[:, :, None]
        ps = (sa[near, None] + q * (sb - sa)[near, None])[:, None]
        closest = float((pr - ps).norm(dim=3).min())
    fine = max(2, math.ceil(longest / closest))           # panels no longer than the closest pair's distance
    for ids, (x, w) in (((far & ~touch).nonzero()[:, 0], _gauss(1, 10 + int(reach))), (near, _gauss(fine, 16))):
        for part in ids.split(max(1, (1 << 24) // len(x) ** 2)):
            pr = ra[part, None] + x[:, None] * (rb - ra)[part, None]
            ps = sa[part, None] + x[:, None] * (sb - sa)[part, None]
            r = torch.zeros((len(part), len(x), len(x)), dtype=torch.float64, device=DEV)
            for c in range(3):
                r += (pr[:, :, None, c] - ps[:, None, :, c]) ** 2
            r = r.sqrt()
            f = w[:, None] * w / r
            for k in range(len(g)):
                out[part, k] = (torch.exp(-g[k] * r) * f).sum(dim=(1, 2))
    return out


def _impedances(elec, img, s, kappa):
    """ZL, ZT (samples, m, m) with images, ref_l = 1."""
    m = len(elec)
    gamma = np.sqrt(s * tags.MU0 * kappa)
    ref_t = _t((kappa - s * tags.EPS0) / (kappa + s * tags.EPS0))
    k, i = np.tril_indices(m)                          # receiver k >= sender i
    d = elec[:, 3:6] - elec[:, :3]
    c_l, c_t = _t(s * tags.MU0 / tags.FOUR_PI), _t(1 / (tags.FOUR_PI * kappa))
    zl = torch.zeros((len(s), m, m), dtype=torch.complex128, device=DEV)
    zt = torch.zeros_like(zl)
    off = k != i
    ti, tk = _t(i), _t(k)
    for other, direct in ((elec, True), (img, False)):
        ii, kk = (i[off], k[off]) if direct else (i, k)
        ti, tk = _t(ii), _t(kk)
        j = _pair_integrals(other[kk], elec[ii], gamma)
        cost = np.abs(np.sum(d[ii] * (other[kk, 3:6] - other[kk, :3]), axis=1))
        fac = _t(np.where(cost > 2.220446049250313e-16, cost, 0.0))
        zl[:, tk, ti] += (c_l[None, :] * j * fac[:, None]).T
        zt[:, tk, ti] += ((c_t if direct else c_t * ref_t)[None, :] * j).T
    ln, k1 = elec[:, 9], elec[:, 10] / elec[:, 9]
    k2 = np.sqrt(1 + k1 * k1)
    self_ = _t(2 * ln * (np.log((k2 + 1) / k1) - k2 + k1))
    q = torch.arange(m, device=DEV)
    zl[:, q, q] += c_l[:, None] * self_
    zt[:, q, q] += c_t[:, None] * self_ / _t(ln * ln)
    low = torch.tril(torch.ones((m, m), dtype=torch.bool, device=DEV), -1)
    for z in (zl, zt):
        z += torch.where(low, z, torch.zeros_like(z)).transpose(1, 2).clone()
    return zl, zt


def _incidence(elec, nodes):
    near = lambda p: np.all(np.abs(p[:, None] - nodes[None]) < 1e-5, axis=2)      # noqa: E731
    start, end = near(elec[:, :3]), near(elec[:, 3:6])
    a = np.where(start, 1.0, np.where(end, -1.0, 0.0))
    return _t(a + 0j), _t(np.where(start | end, 0.5, 0.0) + 0j)                      # m x n


def _solutions(zl, zt, a, b, inj):
    """[U; I_L; I_T] by the node block's Schur complement, one solve per sample."""
    out = []
    for q in range(len(zl)):
        ya, yb = torch.linalg.solve(zl[q], a), torch.linalg.solve(zt[q], b)
        y = a.T @ ya + b.T @ yb
        rhs = torch.zeros(y.shape[0], dtype=torch.complex128, device=DEV)
        rhs[inj] = 1.0
        u = torch.linalg.solve(y, rhs)
        out.append(torch.cat([u, ya @ u, yb @ u]))
    return torch.stack(out)


def _exact_solutions(elec, img, nodes, s, kappa, inj):
    a, b = _incidence(elec, nodes)
    m = len(elec)
    step, out = max(1, int(1.5e9 / (64 * m * m))), []
    for q in range(0, len(s), step):
        zl, zt = _impedances(elec, img, s[q:q + step], kappa[q:q + step])
        out.append(_solutions(zl, zt, a, b, inj))
        del zl, zt
    return torch.cat(out).cpu().numpy()


def _point_sums(points, d, want_field):
    """pot (ns, P, nrhs), vec and field (ns, P, nrhs, 3) at the points."""
    elec = d["elec"]
    x, w = _gauss(max(4, math.ceil(elec[:, 9].max() / 0.5)), 16)     # panels no longer than the points' distance
    a, dv, pts = _t(elec[:, :3]), _t(elec[:, 3:6] - elec[:, :3]), _t(points)
    il, it, g, kap = (_t(d[v]) for v in ("il", "it", "gamma", "kappa"))
    ns, nrhs, _ = il.shape
    pot = torch.zeros((ns, len(points), nrhs), dtype=torch.complex128, device=DEV)
    vec, ef = (torch.zeros((ns, len(points), nrhs, 3), dtype=torch.complex128, device=DEV) for _ in range(2))
    src = a[:, None] + x[:, None] * dv[:, None]                                     # m, q, 3
    step = max(1, (1 << 23) // (len(elec) * len(x)))
    for p0 in range(0, len(points), step):
        sl = slice(p0, p0 + step)
        dx = pts[sl, None, None] - src[None]
        r = dx.norm(dim=3)
        f, f3 = w / r, (w / r ** 3)[..., None] * dx
        for k in range(ns):
            e = torch.exp(-g[k] * r)
            u = (e * f).sum(dim=2)                                                   # P, m
            pot[k, sl] = (u @ it[k].T) / (tags.FOUR_PI * kap[k])
            for c in range(3):
                vec[k, sl, :, c] = (u @ (il[k] * dv[:, c]).T) * (tags.MU0 / tags.FOUR_PI)
            if want_field:
                e = (1 + g[k] * r) * e
                for c in range(3):
                    ef[k, sl, :, c] = ((e * f3[..., c]).sum(dim=2) @ it[k].T) / (tags.FOUR_PI * kap[k])
    return pot, vec, ef


def exact(case, seed):
    d = _inputs(case, seed)
    kind = case["kind"]
    if kind == "plan":
        m, n = _sizes(case)
        if case["ns"] * (m * m * 400.0 + 8.0 * (m + n) ** 3 / 3 + 3e6) > 1.5e12:
            return None
        return {"sol": _exact_solutions(d["elec"], d["img"], d["nodes"], d["s"], d["kappa"], d["inj"]), "info": None}
    if kind == "grids":
        if sum(len(j["electrodes"]) ** 3 for j in d["jobs"]) * case["ns"] > 4e10:
            return None
        return [{"sol": _exact_solutions(j["electrodes"], j["images"], j["nodes"], j["s"], j["kappa"], 0),
                 "info": None} for j in d["jobs"]]
    if kind == "dropin":
        zl, zt = _impedances(d["elec"], d["img"], d["s"], d["kappa"])
        x = _solutions(zl, zt, *_incidence(d["elec"], d["nodes"]), d["inj"])[0]
        # column-major lower triangles: column i from row i on
        tri = [torch.tril(z[0]).T.reshape(-1).cpu().numpy() for z in (zl, zt)]
        return {"zl": tri[0], "zt": tri[1], "x": x.cpu().numpy(), "rc": None}
    if kind == "admittance":
        m, n = len(d["elec"]), len(d["nodes"])
        zl, zt = (np.tril(z.reshape(m, m).T) for z in _mhem_potentials(d))
        zl, zt = (_t(z + np.tril(z, -1).T) for z in (zl, zt))
        a, b = _incidence(d["elec"], d["nodes"])
        ya, yb = torch.linalg.solve(zl, a), torch.linalg.solve(zt, b)
        y = a.T @ ya + b.T @ yb
        rhs = torch.zeros(n, dtype=torch.complex128, device=DEV)
        rhs[d["inj"]] = 1.0
        flat = lambda v: v.T.reshape(-1).cpu().numpy()                               # noqa: E731
        return {"yla": flat(ya), "ytb": flat(yb), "yn": flat(y), "x": torch.linalg.solve(y, rhs).cpu().numpy(),
                "rc": None}
    if kind == "fields":
        pot, vec, ef = _point_sums(d["points"], d, True)
        return {"pot": pot.cpu().numpy(), "vecpot": vec.cpu().numpy(), "efield": ef.cpu().numpy(), "status": None}
    if kind == "voltage":
        p1, p2 = d["paths"][:, :3], d["paths"][:, 3:]
        pot, _, _ = _point_sums(np.concatenate([p1, p2]), d, False)
        length = np.linalg.norm(p2 - p1, axis=1)
        np_ = len(p1)
        out = (pot[:, :np_] - pot[:, np_:]) / _t(length)[None, :, None]
        x, w = np.polynomial.legendre.leggauss(32)
        unit = _t((p2 - p1) / length[:, None])
        for xq, wq in zip(0.5 * (x + 1), 0.5 * w):      # the inductive part along the path
            _, vec, _ = _point_sums(p1 + xq * (p2 - p1), d, False)
            out -= wq * _t(d["s"])[:, None, None] * (vec * unit[None, :, None, :]).sum(dim=3)
        return out.cpu().numpy()
    nt, s, filt = d["nt"], d["s"], d["filter"]
    q = s.imag / s[-1].imag
    sigma = {0: 1.0 + 0 * q, 1: 0.42 + 0.5 * np.cos(math.pi * q) + 0.08 * np.cos(2 * math.pi * q),
             2: (1 + np.cos(math.pi * q)) / 2, 4: 1 - q * q}[filt]
    dt = d["tmax"] / (nt - 1)
    y = np.fft.irfft(sigma[:, None] * d["g"], n=nt, axis=0)
    return y * (np.exp(s[0].real * dt * np.arange(nt)) / dt)[:, None]
