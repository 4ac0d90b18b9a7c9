"""The mixed form's failure paths, driven without faulting or hanging the GPU.

* Refinement that does not converge: a cap of one refinement step
  (tags_plan_set_max_steps) leaves every sample unconverged, so each is
  re-solved by the plain FP64 path (partial pivoting).
* A tensor-core wait that runs out: the waits of the factorisation kernels'
  main loops are limited to 1 ns (tags_debug_tc_wait_limit), so the first
  wait not satisfied at once gives up. The kernel raises its error word, lets
  the copies and products it issued finish (those waits keep their 50 ms
  limit), frees its tensor memory and returns; the pass is re-solved in FP64.
Both must return the plain FP64 solution, and the plan must work normally
afterwards."""
import numpy as np
import pytest

from conftest import golden, rel_err

pytestmark = pytest.mark.gpu


def _case(pkg, count=16):
    gd = golden("grid2.npz")
    e, nodes = gd["elec"], gd["nodes"]
    idx = np.linspace(0, len(gd["s"]) - 1, count).astype(int)
    s, kappa = gd["s"][idx], gd["kappa"][idx]
    ie = np.zeros((count, nodes.shape[0]), np.complex128)
    ie[:, 0] = gd["inj_s"][idx]
    plain, info, _ = pkg.hem_sweep(e, pkg.images(e), nodes, s, kappa, ie=ie, precision=pkg.PLAIN_FP64)
    assert np.all(info == 0)
    return e, nodes, s, kappa, ie, plain


@pytest.mark.parametrize("graphs", [True, False])
def test_refinement_cap_sends_samples_to_fp64(gpu_pkg, graphs):
    pkg = gpu_pkg
    e, nodes, s, kappa, ie, plain = _case(pkg)
    n = nodes.shape[0]
    plan = pkg.Plan(e, pkg.images(e), nodes, pkg.MIXED, max_batch=16, graphs=graphs)
    try:
        plan.set_max_steps(1)
        sol, info, st = plan.run(s, kappa, 1.0, ie)
        assert np.all(info == 0)
        assert st.fallbacks == len(s)
        assert rel_err(sol, plain) < 1e-10
        plan.set_max_steps(0)
        sol, info, st = plan.run(s, kappa, 1.0, ie)
        assert np.all(info == 0) and st.fallbacks == 0
        assert rel_err(sol[:, :n], plain[:, :n]) < 1e-6
    finally:
        plan.close()


def test_tensor_core_wait_expiry_falls_back_to_fp64(gpu_pkg):
    pkg = gpu_pkg
    e, nodes, s, kappa, ie, plain = _case(pkg)
    n = nodes.shape[0]
    plan = pkg.Plan(e, pkg.images(e), nodes, pkg.MIXED, max_batch=16)
    try:
        pkg.lib().tags_gpu_set_quiet(1)
        pkg.debug_tc_wait_limit(1)
        try:
            sol, info, st = plan.run(s, kappa, 1.0, ie)
        finally:
            pkg.debug_tc_wait_limit(0)
            pkg.lib().tags_gpu_set_quiet(0)
        assert "timeout" in pkg.last_error()
        assert np.all(info == 0)
        assert st.fallbacks == len(s)
        assert rel_err(sol, plain) < 1e-10
        # the limit restored, the same plan factorises on the tensor cores again
        sol, info, st = plan.run(s, kappa, 1.0, ie)
        assert np.all(info == 0) and st.fallbacks == 0
        assert rel_err(sol[:, :n], plain[:, :n]) < 1e-6
    finally:
        plan.close()


def test_invalid_samples_are_reported_and_the_plan_recovers(gpu_pkg):
    """A NaN Laplace sample from host memory is refused before any launch
    (TAGS_E_NONFINITE). From device memory it reaches the coefficient kernel,
    which reports it and hands the fill finite coefficients instead, so no
    quadrature order is derived from a NaN; a finite |gamma| beyond 1e5 / m is
    reported the same way (TAGS_E_ARG). The plan keeps its fp16 split and
    solves the next run normally."""
    torch = pytest.importorskip("torch")
    pkg = gpu_pkg
    e, nodes, s, kappa, ie, plain = _case(pkg)
    n, N = nodes.shape[0], plain.shape[1]
    plan = pkg.Plan(e, pkg.images(e), nodes, pkg.MIXED, max_batch=16)
    pkg.lib().tags_gpu_set_quiet(1)
    try:
        bad = s.copy()
        bad[3] = complex(np.nan, 0.0)
        with pytest.raises(RuntimeError, match=f"failed \\({pkg.E_NONFINITE}\\)"):
            plan.run(bad, kappa, 1.0, ie)
        dev = torch.device("cuda", 0)
        k_d = torch.from_numpy(kappa).to(dev)
        ie_d = torch.from_numpy(ie).to(dev)
        sol_d = torch.empty((len(s), N), dtype=torch.complex128, device=dev)
        info_d = torch.empty((len(s),), dtype=torch.int32, device=dev)
        for value, code in ((complex(np.nan, 0.0), pkg.E_NONFINITE), (complex(0.0, 1e20), pkg.E_ARG)):
            bad = s.copy()
            bad[5] = value
            s_d = torch.from_numpy(bad).to(dev)
            with pytest.raises(RuntimeError, match=f"failed \\({code}\\)"):
                plan.run_device(s_d.data_ptr(), k_d.data_ptr(), len(s), 1.0, ie_d.data_ptr(), 0, sol_d.data_ptr(),
                                info_d.data_ptr())
            torch.cuda.synchronize()
    finally:
        pkg.lib().tags_gpu_set_quiet(0)
    try:
        sol, info, st = plan.run(s, kappa, 1.0, ie)
        assert np.all(info == 0) and st.fallbacks == 0
        assert st.split == 16                       # the NaN did not switch the plan to bf16 pieces
        assert rel_err(sol[:, :n], plain[:, :n]) < 1e-6
    finally:
        plan.close()


def test_memory_budget_below_one_sample_reports_nomem(gpu_pkg):
    """With the process-wide memory budget below what one sample needs, a new
    plan fails with TAGS_E_NOMEM (nothing is left allocated); with the budget
    lifted the same plan builds and solves."""
    pkg = gpu_pkg
    e, nodes, s, kappa, ie, plain = _case(pkg, 4)
    n = nodes.shape[0]
    pkg.lib().tags_gpu_set_quiet(1)
    pkg.set_memory_budget(1 << 20)
    try:
        with pytest.raises(RuntimeError, match=f"failed \\({pkg.E_NOMEM}\\)"):
            pkg.Plan(e, pkg.images(e), nodes, pkg.MIXED)
    finally:
        pkg.set_memory_budget(0)
        pkg.lib().tags_gpu_set_quiet(0)
    plan = pkg.Plan(e, pkg.images(e), nodes, pkg.MIXED)
    try:
        sol, info, st = plan.run(s, kappa, 1.0, ie)
        assert np.all(info == 0)
        assert rel_err(sol[:, :n], plain[:, :n]) < 1e-6
    finally:
        plan.close()


@pytest.mark.parametrize("m,ns", [(7, 1), (7, 70), (21, 65), (40, 33), (107, 3)])
def test_resolves_side_by_side_match_plain(gpu_pkg, m, ns):
    """Every sample re-solved in FP64 (one refinement step allowed), several at
    a time (at most 64) and over both forms of the structured solve, with one
    sample (s = 0) that needs the pivoted LU: equal to the plain form."""
    pkg = gpu_pkg
    z = -0.6 - 0.7 * np.arange(m + 1)
    nodes = np.stack([0.5 * (np.arange(m + 1) % 2), np.zeros(m + 1), z], axis=1)
    e = np.stack([pkg.populate_electrode(nodes[i], nodes[i + 1], 7e-3) for i in range(m)])
    img = pkg.images(e)
    s = 8e4 + 2j * np.pi * np.linspace(1e4, 5e6, ns)
    kappa = 0.004 + s * 10 * pkg.EPS0
    if ns > 2:
        s[1], kappa[1] = 0.0, 0.004
    ref, info, _ = pkg.hem_sweep(e, img, nodes, s, kappa, inj_node=1)
    assert not info.any()
    plan = pkg.Plan(e, img, nodes, pkg.MIXED, ns)
    try:
        plan.set_max_steps(1)
        sol, info, st = plan.run(s, kappa, inj_node=1)
        assert st.fallbacks == ns and not info.any()
        assert np.max(np.abs(sol - ref)) < 1e-10 * np.max(np.abs(ref))
    finally:
        plan.close()


@pytest.mark.parametrize("m", [6, 40, 120])
@pytest.mark.parametrize("value,kappa_value", [(complex(np.nan, 0.0), 0.01 + 1e-4j), (complex(0.0, 1e20), 0.01 + 1e-4j)])
def test_samples_beside_an_invalid_one_are_solved(gpu_pkg, m, value, kappa_value):
    """A plain run with an invalid sample fails, and its other samples are
    solved all the same, those of s = 0 that need the pivoted LU among them, in
    the pass of the invalid one and in later ones: equal to a run without it.
    info holds 0 or a pivot's number, never an internal mark, also after a
    geometry error."""
    torch = pytest.importorskip("torch")
    pkg = gpu_pkg
    e, nodes = pkg.segment_electrode([0.0, 0.0, -0.5], [1.0 * m, 0.0, -0.5], m, 7e-3)
    s = np.array([8e4 + 1e5j, 0.0, 8e4 + 1e6j, value, 0.0, 8e4 + 2e6j, 0.0])
    kappa = np.where(s == 0.0, 0.01 + 0j, 0.01 + 1e-4j)
    kappa[3] = kappa_value
    good = np.array([0, 1, 2, 4, 5, 6])
    want, info, _ = pkg.hem_sweep(e, pkg.images(e), nodes, s[good], kappa[good], inj_node=1)
    assert not info.any()
    pkg.lib().tags_gpu_set_quiet(1)
    try:
        for case in ("invalid sample", "geometry"):
            es = e if case == "invalid sample" else np.concatenate([e, e[:1]])
            for graphs in (True, False):
                plan = pkg.Plan(es, pkg.images(es), nodes, pkg.PLAIN_FP64, 5, graphs)
                s_d, k_d = (torch.from_numpy(v).cuda() for v in (s, kappa))
                sol = torch.zeros((len(s), plan.N), dtype=torch.complex128, device="cuda")
                got = torch.full((len(s),), 77, dtype=torch.int32, device="cuda")
                try:
                    with pytest.raises(RuntimeError):
                        plan.run_device(s_d.data_ptr(), k_d.data_ptr(), len(s), 1.0, 0, 1, sol.data_ptr(), got.data_ptr())
                finally:
                    plan.close()
                torch.cuda.synchronize()
                assert not got.cpu().numpy()[good].any()
                if case == "invalid sample":
                    assert rel_err(sol.cpu().numpy()[good], want) < 1e-10
        if np.isfinite(value):                      # a grid batch takes finite values only
            jobs = [{"electrodes": e, "images": pkg.images(e), "nodes": nodes, "s": s, "kappa": kappa, "inj_node": 1}]
            batch = pkg.GridBatch(jobs, precision=pkg.PLAIN_FP64)
            try:
                arr, keep, out = pkg._grid_jobs(jobs)
                assert pkg.lib().tags_batch_run(batch.handle, arr, 1, None) == pkg.E_ARG
            finally:
                batch.close()
            assert not out[0][1][good].any()
            assert rel_err(out[0][0][good], want) < 1e-10
    finally:
        pkg.lib().tags_gpu_set_quiet(0)


@pytest.mark.parametrize("gap", [0.0, 700.0])
def test_plain_plans_keep_to_the_share_of_memory_they_size_for(gpu_pkg, gap):
    """Plans take at most 0.45 of the free memory for their samples and grid batches 0.6, the fill's tables included,
    which for two segments far apart are 16 KB a sample beside a matrix of 1 KB."""
    torch = pytest.importorskip("torch")
    pkg = gpu_pkg
    ends = [((gap * i, 0.3 * i, -0.5), (gap * i, 0.3 * i, -1.5)) for i in range(2)]
    e = np.stack([pkg.populate_electrode(a, b, 7e-3) for a, b in ends])
    nodes = np.array([p for pair in ends for p in pair])
    s, budget = 8e4 + 2j * np.pi * np.linspace(1e3, 1e5, 60000), 1 << 30
    kappa = np.full(len(s), 0.01 + 1e-4j)
    jobs = [{"electrodes": e, "images": pkg.images(e), "nodes": nodes, "s": s, "kappa": kappa, "inj_node": 0}]
    pkg.hem_sweep(e, pkg.images(e), nodes, s[:2], kappa[:2])
    pkg.set_memory_budget(budget)
    try:
        for share, make in ((0.45, lambda: pkg.Plan(e, pkg.images(e), nodes, pkg.PLAIN_FP64, 60000)),
                            (0.60, lambda: pkg.GridBatch(jobs, precision=pkg.PLAIN_FP64, max_batch=60000))):
            before = torch.cuda.mem_get_info()[0]
            held = make()
            try:
                assert before - torch.cuda.mem_get_info()[0] <= share * budget + (24 << 20)
            finally:
                held.close()
    finally:
        pkg.set_memory_budget(0)


def test_path_voltages_without_room_for_their_tables(gpu_pkg):
    """With too little device memory left for the pair integrals' tables (0.66 GB here) the call takes the rule per
    sample, which needs none: the same voltages to the two rules' agreement of 1e-12, not an allocation error."""
    torch = pytest.importorskip("torch")
    pkg = gpu_pkg
    e = np.stack([pkg.populate_electrode([700.0 * i, 0, -0.5], [700.0 * i, 0, -1.5], 7e-3) for i in range(2)])
    ns = 40000
    cur = np.ones((ns, 1, 2), np.complex128)
    args = (np.array([[5.0, 1, 0, 6.0, 1, 0]]), e, cur, cur, np.full(ns, 0.01 + 0.01j), np.full(ns, 1e5j),
            np.ones(ns, np.complex128))
    few = [a if k < 2 else a[:3] for k, a in enumerate(args)]
    want = pkg.voltage_batch(*few)
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - (400 << 20), dtype=torch.uint8, device="cuda")
    try:
        got = pkg.voltage_batch(*args)
    finally:
        del held
        torch.cuda.empty_cache()
    assert rel_err(got, np.broadcast_to(want[:1], got.shape)) < 1e-12


def test_resolves_buffer_grows_and_stays_when_it_cannot(gpu_pkg):
    """The FP64 re-solves' buffer of a plan: taken for one sample, grown for more, and, with no device memory for a larger
    one, kept as it is; the same solutions each time."""
    torch = pytest.importorskip("torch")
    pkg = gpu_pkg
    m, ns = 250, 40                             # 9 MB a sample
    e, nodes = pkg.segment_electrode([0.0, 0.0, -0.5], [1.0 * m, 0.0, -0.5], m, 7e-3)
    s = 8e4 + 2j * np.pi * np.linspace(1e4, 5e6, ns)
    kappa = 0.004 + s * 10 * pkg.EPS0
    want, info, _ = pkg.hem_sweep(e, pkg.images(e), nodes, s, kappa, inj_node=1)
    plan = pkg.Plan(e, pkg.images(e), nodes, pkg.MIXED, ns)
    held = []
    try:
        plan.set_max_steps(1)
        for take in (1, 3, 12, ns):
            plan.run(s[:take], kappa[:take], inj_node=1)          # the pass's graph is built here
            if take == 12:
                torch.cuda.empty_cache()
                held.append(torch.empty(torch.cuda.mem_get_info()[0] - (64 << 20), dtype=torch.uint8, device="cuda"))
            sol, info, st = plan.run(s[:take], kappa[:take], inj_node=1)
            assert st.fallbacks == take and not info.any()
            assert np.max(np.abs(sol - want[:take])) < 1e-10 * np.max(np.abs(want))
    finally:
        plan.close()
        held.clear()
        torch.cuda.empty_cache()
