"""Grids at the edges of the ionosphere solvers' launch shapes: sweep blocks of
64 colatitude rows (tensor solve), column bands of 4 to 16 rows and whole or
partial warps of longitudes (PCG)."""
import ctypes as C

import numpy as np
import pytest

from gamera_cube_b200 import abi, cases
from oracle import oracle_cases

pytestmark = pytest.mark.gpu
D = C.POINTER(C.c_double)


@pytest.fixture(scope="module")
def lib():
    import gamera_cube_b200
    return gamera_cube_b200.lib


def at(a):
    return a.ctypes.data_as(D)


@pytest.mark.parametrize("npl,nt", [
    (18, 65),    # 63 rows: one block, its last row empty
    (18, 66),    # one full block
    (19, 67),    # a second block of one row
    (33, 130),   # two full blocks
    (24, 195),   # a fourth block of one row
    (6, 68),     # head and seam of a row in the same group of steps
    (64, 4),     # two rows
])
def test_tensor_blocks(lib, npl, nt):
    """The one-warp-per-block sweeps (schedule 0) against the oracle: the
    potential within twice the oracle's own 1e-8 error of its 1e-12 solve
    plus 5e-8 of the maximum, the bound of the tall narrow grids."""
    case = cases.mi_case(npl, nt, seed=npl + nt, max_iterations=20000)
    tight = cases.mi_case(npl, nt, seed=npl + nt, max_iterations=200000, rel_tol=1e-12)
    o = oracle_cases.lib()
    got = []
    for cfg in (tight.config, case.config):
        p, st = np.zeros((nt, npl)), abi.MiSolverStats()
        assert o.gcso_mi_solve_conductance_tensor(
            C.byref(cfg), at(case.fac), at(case.pedersen), at(case.hall), at(p),
            C.byref(st)) == 0
        got.append(p)
    truth, ref = got
    plan, st, status = C.c_void_p(), abi.MiSolverStats(), C.c_int()
    assert lib.gcs_mi_tensor_plan_create(C.byref(case.config), C.byref(plan)) == 0
    try:
        assert lib.gcs_mi_tensor_plan_set_schedule(plan, 0) == 0
        pot = np.zeros((nt, npl))
        buffers = [C.c_void_p() for _ in range(4)]
        lib.gcs_mi_tensor_plan_buffers(plan, *[C.byref(b) for b in buffers])
        for _ in range(2):   # the inboxes are left empty for the next solve
            assert lib.gcs_mi_tensor_plan_upload(plan, at(case.fac), at(case.pedersen),
                                                 at(case.hall), at(pot)) == 0
            assert lib.gcs_mi_tensor_solve_async(plan, None) == 0
            assert lib.gcs_mi_tensor_results(plan, C.byref(st), C.byref(status)) == 0
            assert status.value == 0
        import torch

        class View:
            __cuda_array_interface__ = {"shape": (nt, npl), "typestr": "<f8", "version": 3,
                                        "data": (buffers[3].value, False)}
        out = torch.as_tensor(View(), device="cuda").cpu().numpy()
    finally:
        lib.gcs_mi_tensor_plan_destroy(plan)
    scale = np.abs(truth).max()
    assert np.abs(out - truth).max() <= 2.0 * np.abs(ref - truth).max() + 5e-8 * scale


@pytest.mark.parametrize("npl,nt", [(32, 6), (33, 7), (31, 66), (64, 67), (65, 130),
                                    (384, 19), (385, 19), (256, 258), (4, 3)])
@pytest.mark.parametrize("iterations", [1, 4, 12])
@pytest.mark.parametrize("variable", [False, True])
def test_pcg_bands(lib, npl, nt, iterations, variable):
    """The first iterates of both PCG solves against the restatement, to 1e-11
    of the maximum (rounding has not grown by then)."""
    case = cases.mi_case(npl, nt, seed=npl + nt, max_iterations=iterations)
    ped = case.pedersen.copy()
    ped[0, :] = ped[0, :].mean()
    o, out, its = oracle_cases.lib(), [], []
    calls = ((lib.gcs_mi_solve_pedersen_pcg, o.gcso_mi_solve_pedersen_pcg) if variable else
             (lib.gamera_mi_solve_constant_pedersen, o.gcso_mi_solve_constant_pedersen))
    for call in calls:
        p, st = np.zeros((nt, npl)), abi.MiSolverStats()
        args = [at(case.fac)] + ([at(ped)] if variable else []) + [at(p), C.byref(st)]
        call(C.byref(case.config), *args)
        out.append(p)
        its.append(st.iterations)
    assert its[0] == its[1]
    assert np.abs(out[0] - out[1]).max() <= 1e-11 * np.abs(out[1]).max()
