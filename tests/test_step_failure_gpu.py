"""What a failed step reports and leaves behind, on wind cases whose
background field (host arrays of the oracle's case) is made NaN at chosen
faces, edges or cells: a flux, EMF or update failure exactly there."""
import ctypes as C

import numpy as np
import pytest

from gamera_cube_b200 import abi
from oracle import oracle_cases

pytestmark = pytest.mark.gpu

KINETIC_MAXWELL, EDGE_EMF, UPDATE = 5, 11, 12


@pytest.fixture(scope="module")
def lib():
    import gamera_cube_b200
    return gamera_cube_b200.lib


def field(pointer, shape):
    """numpy view of a Vec3 array of a background field."""
    at = C.cast(pointer, C.POINTER(C.c_double))
    return np.ctypeslib.as_array(at, shape=tuple(shape) + (3,))


def failed_step(lib, case):
    """One step that has to fail; (stage, direction, face, (i, j, k))."""
    plan = C.c_void_p()
    assert lib.gamera_cs_halo_plan_create(case.grid, case.active, case.ghost,
                                          C.byref(plan)) == 0, lib.gcs_last_error()
    try:
        dt = 0.4 * case.local_timestep()
        assert lib.gamera_cs_advance_six_with_background_planned(
            case.grid, case.storage, case.active, case.ghost, 0.0, dt, case.options,
            case.background, plan, None, 0.0, 0.0, None) == -1
        v = [C.c_int() for _ in range(5)]
        stage = lib.gcs_context_failure(lib.gcs_halo_plan_context(plan),
                                        *[C.byref(q) for q in v])
        return stage, v[0].value, v[1].value, tuple(q.value for q in v[2:])
    finally:
        lib.gamera_cs_halo_plan_destroy(plan)


@pytest.fixture(scope="module")
def case():
    c = oracle_cases.Case("wind", 24, 12, 3)
    yield c
    c.close()


@pytest.mark.parametrize("family", ["flux", "emf"])
def test_first_failure_is_of_the_lowest_direction(lib, case, family):
    """The directions of a sweep run in one launch: of failures of several
    directions the lowest direction's lowest face, layer and index is
    reported, not the first that a block met.  The higher directions fail on
    the first face and layer, direction 0 on the last."""
    g, (nr, n) = case.ghost, list(case.active)[:2]
    ext = [nr + 2 * g, n + 2 * g, n + 2 * g]
    kept = []
    for d, face, cell in [(2, 0, (g, g, g)), (1, 0, (g, g + 1, g)), (1, 1, (g, g, g)),
                          (0, 5, (g + nr - 1, g + n - 1, g + n - 1)),
                          (0, 5, (g + nr - 1, g + n - 2, g + n - 1))]:
        bg = case.background[face]
        if family == "flux":
            at = field(bg.face_magnetic[d], [e + (a == d) for a, e in enumerate(ext)])
        else:
            at = field(bg.edge_magnetic[d], [e + (a != d) for a, e in enumerate(ext)])
        kept.append((at, cell, at[cell].copy()))
        at[cell] = np.nan
    try:
        stage, d, face, cell = failed_step(lib, case)
    finally:
        for at, cell_, value in kept:
            at[cell_] = value
    assert stage == (KINETIC_MAXWELL if family == "flux" else EDGE_EMF)
    assert (d, face, cell) == (0, 5, (g + nr - 1, g + n - 2, g + n - 1))


@pytest.mark.parametrize("mode", ["drop_in", "step", "run", "run_graph"])
def test_failed_update_leaves_the_field(lib, case, mode):
    """A NaN background force fails the momentum update of one cell: the step
    stops there, and B of every active cell is the one it began with."""
    g, (nr, n) = case.ghost, list(case.active)[:2]
    ext = [nr + 2 * g, n + 2 * g, n + 2 * g]
    act = (slice(g, g + nr), slice(g, g + n), slice(g, g + n))
    cell = (g + 3, g + 5, g + 7)
    force = field(case.background[2].cell_force, ext)
    kept = force[cell].copy()
    before = [case.arrays(f)["cell_magnetic"][act].copy() for f in range(6)]
    force[cell] = np.nan
    try:
        if mode == "drop_in":
            stage, _, face, at = failed_step(lib, case)
        else:
            ctx = lib.gcs_context_create(case.grid, case.active, case.ghost)
            assert ctx, lib.gcs_last_error()
            assert lib.gcs_context_upload_background(ctx, case.background) == 0
            assert lib.gcs_context_upload_state(ctx, case.storage) == 0
            if mode == "step":
                assert lib.gcs_context_step(ctx, case.options, 0.0,
                                            0.4 * case.local_timestep()) == -1
            else:
                assert lib.gcs_context_run(ctx, case.options, case.timestep_options, 0.5, 3,
                                           int(mode == "run_graph")) == 0
                assert lib.gcs_context_sync(ctx) == -1
            v = [C.c_int() for _ in range(5)]
            stage = lib.gcs_context_failure(ctx, *[C.byref(q) for q in v])
            face, at = v[1].value, tuple(q.value for q in v[2:])
            assert lib.gcs_context_download_state(ctx, case.storage, 0) == 0
            lib.gcs_context_destroy(ctx)
    finally:
        force[cell] = kept
    assert (stage, face, at) == (UPDATE, 2, cell)
    for f in range(6):
        now = case.arrays(f)["cell_magnetic"][act]
        np.testing.assert_array_equal(now, before[f])
