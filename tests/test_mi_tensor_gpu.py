"""The CUDA conductance-tensor solve (SSOR-BiCGStab) against the
reference.  The BiCGStab dot products are summed in a fixed parallel order,
so iterates differ from the CPU solver's at rounding level; a solve passes
when it converges, its true residual -- evaluated on the CPU with the
oracle's tensor operator -- meets the reference target (slack 1e-9), its
potential is within 5e-8 of max|potential| of the reference's and its
iteration count within 10 % (at least 3)."""
import ctypes as C

import numpy as np
import pytest

from mi_util import POTENTIAL_RTOL, golden, golden_case, ptr
from oracle import oracle_cases

pytestmark = pytest.mark.gpu


def glib():
    import gamera_cube_b200
    return gamera_cube_b200.lib


def tensor_residual(cfg, fac, sp, sh, pot):
    npl, nt = cfg.longitude_count, cfg.colatitude_count
    ap = np.zeros_like(pot)
    assert oracle_cases.lib().gcso_mi_apply_conductance_tensor(
        C.byref(cfg), ptr(sp), ptr(sh), ptr(pot), ptr(ap)) == 0
    dth = cfg.maximum_colatitude / (nt - 1)
    th = dth * np.arange(1, nt - 1)
    c = np.cos(th)
    inc = cfg.hemisphere * 2.0 * c / np.sqrt(1.0 + 3.0 * c * c)
    u = -(cfg.ionosphere_radius_m ** 2) * fac[1:nt - 1] * inc[:, None]
    res = u - ap[1:nt - 1]
    # pole row: the reduced system's pole equation, scaled like the reference norm
    norm2 = npl * ap[0, 0] ** 2 + np.sum(res * res)
    target = max(cfg.absolute_tolerance,
                 cfg.relative_tolerance * max(np.sqrt(np.sum(u * u)), 1.0))
    return float(np.sqrt(norm2)), float(target)


def solve(lib, fn, cfg, d, guess):
    from gamera_cube_b200 import abi
    pot = guess.copy()
    st = abi.MiSolverStats()
    rc = fn(C.byref(cfg), ptr(d["fac"]), ptr(d["pedersen"]), ptr(d["hall"]), ptr(pot),
            C.byref(st))
    return rc, pot, st


def check(cfg, d, pot, st, ref_pot, ref_iters):
    assert st.converged == 1
    scale = np.abs(ref_pot).max()
    assert np.abs(pot - ref_pot).max() <= POTENTIAL_RTOL * scale
    assert abs(st.iterations - ref_iters) <= max(3, 0.1 * ref_iters)
    assert np.all(pot[0] == pot[0, 0]) and np.all(pot[-1] == 0.0)


@pytest.mark.parametrize("name", ["small_north", "shell_192x22"])
def test_tensor_against_golden(name):
    g = golden()
    cfg, d = golden_case(g, name, tensor=True)
    rc, pot, st = solve(glib(), glib().gamera_mi_solve_conductance_tensor, cfg, d,
                        d["guess"])
    assert rc == 0
    check(cfg, d, pot, st, g[name + "/tensor/potential"],
          int(g[name + "/tensor/stats"][0]))
    assert st.initial_residual == pytest.approx(g[name + "/tensor/stats"][1], rel=1e-12)


def test_tensor_production_grid():
    """181 x 361, Hall = 1.5 Pedersen, against the oracle."""
    from gamera_cube_b200 import cases
    case = cases.mi_case(361, 181, seed=21, max_iterations=20000)
    d = {"fac": case.fac, "pedersen": case.pedersen, "hall": case.hall}
    O = oracle_cases.lib()
    rc, ref_pot, ref_st = solve(O, O.gcso_mi_solve_conductance_tensor, case.config, d,
                                case.potential)
    assert rc == 0
    rc, pot, st = solve(glib(), glib().gamera_mi_solve_conductance_tensor, case.config,
                        d, case.potential)
    assert rc == 0
    check(case.config, d, pot, st, ref_pot, ref_st.iterations)


@pytest.mark.parametrize("npl,nt,hemisphere", [
    (8, 12, 1),     # bands of one row
    (5, 40, -1),    # bands of three rows, southern hemisphere
    (12, 70, 1),    # bands of five rows
    (9, 35, 1),
    (16, 300, -1),  # the widest grid that starts with bands, of 19 rows
    (17, 60, 1),    # the narrowest grid that starts with row blocks: one
    (40, 250, -1),  # four blocks
    (40, 100, 1),   # two blocks
    (35, 34, -1),   # half a block
])
def test_tensor_grid_shapes(npl, nt, hemisphere):
    """Both sweep schedules, as plans start with them, against the oracle.

    On these tall, narrow grids two solves that each reach relative residual
    1e-8 differ by up to 9e-8 of max|potential| (the reference's own 1e-8
    solution against its 1e-12 one), so the GPU solution is held to the
    reference's accuracy instead: its distance to the oracle's 1e-12 solve
    is at most twice the oracle's 1e-8 solve's, plus 5e-8 of max."""
    from gamera_cube_b200 import cases
    case = cases.mi_case(npl, nt, seed=npl + nt, hemisphere=hemisphere,
                         max_iterations=20000)
    tight = cases.mi_case(npl, nt, seed=npl + nt, hemisphere=hemisphere,
                          max_iterations=200000, rel_tol=1e-12)
    d = {"fac": case.fac, "pedersen": case.pedersen, "hall": case.hall}
    O = oracle_cases.lib()
    rc, truth, _ = solve(O, O.gcso_mi_solve_conductance_tensor, tight.config, d,
                         case.potential)
    assert rc == 0
    rc, ref_pot, ref_st = solve(O, O.gcso_mi_solve_conductance_tensor, case.config, d,
                                case.potential)
    assert rc == 0
    rc, pot, st = solve(glib(), glib().gamera_mi_solve_conductance_tensor, case.config,
                        d, case.potential)
    assert rc == 0, glib().gcs_last_error().decode()
    assert st.converged == 1
    scale = np.abs(truth).max()
    ref_err = np.abs(ref_pot - truth).max()
    assert np.abs(pot - truth).max() <= 2.0 * ref_err + POTENTIAL_RTOL * scale
    assert abs(st.iterations - ref_st.iterations) <= max(3, 0.1 * ref_st.iterations)
    assert np.all(pot[0] == pot[0, 0]) and np.all(pot[-1] == 0.0)


def test_tensor_rejects_bad_input():
    from gamera_cube_b200 import abi, cases
    L = glib()
    case = cases.mi_case(24, 12, seed=3)
    d = {"fac": case.fac.copy(), "pedersen": case.pedersen.copy(),
         "hall": case.hall.copy()}
    d["fac"][4, 5] = np.nan
    pot = np.full_like(case.fac, 2.0)
    st = abi.MiSolverStats()
    st.iterations = -3
    assert L.gamera_mi_solve_conductance_tensor(
        C.byref(case.config), ptr(d["fac"]), ptr(d["pedersen"]), ptr(d["hall"]),
        ptr(pot), C.byref(st)) == -1
    assert np.all(pot == 2.0) and st.iterations == -3
    d["fac"][4, 5] = 0.0
    d["pedersen"][0, 0] = -1.0
    assert L.gamera_mi_solve_conductance_tensor(
        C.byref(case.config), ptr(d["fac"]), ptr(d["pedersen"]), ptr(d["hall"]),
        ptr(pot), C.byref(st)) == -1
    d["pedersen"][0, 0] = 1.0
    bad = cases.mi_config(24, 12, low_latitude_potential_v=3.0)
    assert L.gamera_mi_solve_conductance_tensor(
        C.byref(bad), ptr(d["fac"]), ptr(d["pedersen"]), ptr(d["hall"]), ptr(pot),
        C.byref(st)) == -1


def plan_solve(case, colored, banded=None):
    """The device tensor plan with the given SSOR ordering (and sweep
    schedule, when given); returns the potential, stats, status and device
    milliseconds of one solve."""
    import torch
    from gamera_cube_b200 import abi
    L = glib()
    cudart = C.CDLL("libcudart.so.12")
    plan = C.c_void_p()
    assert L.gcs_mi_tensor_plan_create(C.byref(case.config), C.byref(plan)) == 0
    try:
        assert L.gcs_mi_tensor_plan_set_ordering(plan, colored) == 0
        if banded is not None:
            assert L.gcs_mi_tensor_plan_set_schedule(plan, banded) == 0
        pot = case.potential.copy()
        assert L.gcs_mi_tensor_plan_upload(plan, ptr(case.fac), ptr(case.pedersen),
                                           ptr(case.hall), ptr(pot)) == 0
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s = torch.cuda.current_stream()
        a.record(s)
        assert L.gcs_mi_tensor_solve_async(plan, C.c_void_p(s.cuda_stream)) == 0
        b.record(s)
        st, status = abi.MiSolverStats(), C.c_int()
        assert L.gcs_mi_tensor_results(plan, C.byref(st), C.byref(status)) == 0
        b.synchronize()
        bufs = [C.c_void_p() for _ in range(4)]
        assert L.gcs_mi_tensor_plan_buffers(plan, *[C.byref(x) for x in bufs]) == 0
        host = np.zeros(case.potential.shape)
        assert cudart.cudaMemcpy(C.c_void_p(host.ctypes.data),
                                 bufs[3], C.c_size_t(host.nbytes),
                                 2) == 0
        return host, st, status.value, a.elapsed_time(b)
    finally:
        L.gcs_mi_tensor_plan_destroy(plan)


@pytest.mark.parametrize("npl,nt,hemisphere", [
    (361, 181, 1),   # production grid, odd longitude count (seam colours)
    (40, 250, -1),
    (12, 70, 1),
    (8, 12, 1),
])
def test_colored_ordering_converges_to_the_reference_solution(npl, nt, hemisphere):
    """The multicolour SSOR ordering: converged, and as close to the
    oracle's 1e-12 solve as the reference's own 1e-8 solve is (see
    test_tensor_grid_shapes); iteration count and time recorded."""
    from gamera_cube_b200 import cases
    case = cases.mi_case(npl, nt, seed=npl + nt, hemisphere=hemisphere,
                         max_iterations=20000)
    tight = cases.mi_case(npl, nt, seed=npl + nt, hemisphere=hemisphere,
                          max_iterations=200000, rel_tol=1e-12)
    d = {"fac": case.fac, "pedersen": case.pedersen, "hall": case.hall}
    O = oracle_cases.lib()
    rc, truth, _ = solve(O, O.gcso_mi_solve_conductance_tensor, tight.config, d,
                         case.potential)
    assert rc == 0
    rc, ref, ref_st = solve(O, O.gcso_mi_solve_conductance_tensor, case.config, d,
                            case.potential)
    assert rc == 0
    pot, st, status, ms = plan_solve(case, 1)
    assert status == 0 and st.converged == 1, (status, st.iterations)
    scale = np.abs(truth).max()
    ref_err = np.abs(ref - truth).max()
    assert np.abs(pot - truth).max() <= 2.0 * ref_err + 5e-8 * scale
    # as converged as the reference's own 1e-8 solve, in one residual norm
    res, _ = tensor_residual(case.config, case.fac, case.pedersen, case.hall, pot)
    ref_res, _ = tensor_residual(case.config, case.fac, case.pedersen, case.hall, ref)
    assert res <= 2.0 * ref_res, (res, ref_res)
    print("colored %dx%d: %d iterations (reference ordering %d), %.2f ms"
          % (nt, npl, st.iterations, ref_st.iterations, ms))


@pytest.mark.parametrize("npl,nt,hemisphere", [
    (361, 181, 1),   # production grid: 15 bands of 12 rows on a 16-CTA cluster
    (40, 250, -1),   # 16 bands of 16 rows (the last of 8)
    (12, 70, 1),     # 14 bands of 5 rows (the last of 3)
    (8, 12, 1),      # 10 rows: 10 bands of one row
    (17, 60, 1),
    (5, 40, -1),
    (40, 100, 1),
])
def test_band_schedule_is_bitwise(npl, nt, hemisphere):
    """The band-pipelined sweeps (each CTA of the cluster sweeps its band of
    rows; edge rows cross between CTAs through distributed shared memory)
    against the wavefront of 64-row blocks: the same operations on the same
    operands, so the potential and the stats must agree bit for bit."""
    from gamera_cube_b200 import cases
    L = glib()
    case = cases.mi_case(npl, nt, seed=npl + nt, hemisphere=hemisphere,
                         max_iterations=20000)
    plan = C.c_void_p()
    assert L.gcs_mi_tensor_plan_create(C.byref(case.config), C.byref(plan)) == 0
    h, n = C.c_int(), C.c_int()
    try:
        # the default: bands below 17 longitudes, row blocks from 17 on
        assert L.gcs_mi_tensor_plan_schedule(plan, None, None) == (1 if npl < 17 else 0)
        assert L.gcs_mi_tensor_plan_set_schedule(plan, 1) == 0
        assert L.gcs_mi_tensor_plan_schedule(plan, C.byref(h), C.byref(n)) == 1
        assert L.gcs_mi_tensor_plan_set_schedule(plan, 0) == 0
        assert L.gcs_mi_tensor_plan_schedule(plan, C.byref(h), C.byref(n)) == 0
        assert L.gcs_mi_tensor_plan_set_schedule(plan, 2) == -1
    finally:
        L.gcs_mi_tensor_plan_destroy(plan)
    rows = nt - 2
    assert L.gcs_mi_tensor_plan_create(C.byref(case.config), C.byref(plan)) == 0
    try:
        assert L.gcs_mi_tensor_plan_set_schedule(plan, 1) == 0
        assert L.gcs_mi_tensor_plan_schedule(plan, C.byref(h), C.byref(n)) == 1
    finally:
        L.gcs_mi_tensor_plan_destroy(plan)
    # one band per CTA of the cluster (at most 16), at most 32 rows each
    assert 1 <= h.value <= 32 and n.value == -(-rows // h.value) and n.value <= 16
    pa, sa, ka, ta = plan_solve(case, 0, banded=0)
    pb, sb, kb, tb = plan_solve(case, 0, banded=1)
    assert ka == kb == 0
    assert (sa.iterations, sa.initial_residual, sa.final_residual, sa.converged) == \
        (sb.iterations, sb.initial_residual, sb.final_residual, sb.converged)
    assert np.array_equal(pa, pb)
    print("band schedule %dx%d: row blocks %.2f ms, bands %.2f ms, %d iterations"
          % (nt, npl, ta, tb, sb.iterations))
