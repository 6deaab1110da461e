"""The forms of the step's sweeps and transfers that a plain case does not
reach: face frames that are not orthonormal (the flux sweep then reads the
tangents), the short kernels launched per family, light speeds and layer
counts at the edges, and state transfers at sizes that leave partial blocks
or fail."""
import ctypes as C

import numpy as np
import pytest

from gamera_cube_b200 import abi
from gamera_cube_b200.host import HostStorage
from oracle import oracle_cases
from tests.parity_util import compare_state

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    import gamera_cube_b200
    return gamera_cube_b200.lib


def scale_tangents(case, factor):
    """Tangents of every face times `factor`: the flux projects on them and
    back, so the momentum flux along them scales by factor^2."""
    for f in range(6):
        grid = case.grid[f]
        for d in range(3):
            faces = grid.face[d]
            count = faces.extent[0] * faces.extent[1] * faces.extent[2]
            at = C.cast(faces.value, C.POINTER(C.c_double))
            view = np.ctypeslib.as_array(at, shape=(count, C.sizeof(abi.FaceGeometry) // 8))
            first = abi.FaceGeometry.tangent1.offset // 8
            view[:, first:first + 6] *= factor


@pytest.mark.parametrize("factor", [1.0, 1.0 + 1e-7, 0.9])
@pytest.mark.parametrize("kind,nr,n", [("wind", 12, 9), ("shock", 17, 11)])
def test_frames(lib, kind, nr, n, factor):
    """One step against the restatement on the same grid: 1e-12 normwise,
    orthonormal frames (factor 1) or not.  1e-7 off shows a sweep that took
    the orthonormal form on a frame that is not: the momentum flux along the
    tangents would be 2e-7 off."""
    ref, gpu = oracle_cases.pair(kind, nr, n, 5)
    scale_tangents(ref, factor)
    scale_tangents(gpu, factor)
    plan = C.c_void_p()
    assert lib.gamera_cs_halo_plan_create(gpu.grid, gpu.active, gpu.ghost,
                                          C.byref(plan)) == 0, lib.gcs_last_error()
    try:
        dt = 0.4 * ref.local_timestep()
        assert ref.step(0.0, dt) == 0
        assert lib.gamera_cs_advance_six_with_background_planned(
            gpu.grid, gpu.storage, gpu.active, gpu.ghost, 0.0, dt, gpu.options,
            gpu.background, plan, None, 0.0, 0.0, None) == 0
        bad = {k: v for k, v in compare_state(gpu, ref).items() if not v[0] <= 1e-12}
        assert not bad, bad
    finally:
        lib.gamera_cs_halo_plan_destroy(plan)


@pytest.mark.parametrize("bulk", [0, 1])
def test_one_launch_per_family(lib, bulk):
    """A run of an ensemble (face velocities and CT launched per family, the
    seam sync per time level) and the same run stepped alone (all in a launch)
    agree bit for bit."""
    driver = abi.WindDriver(7.0, -420.0, 9e4, -4.0)
    nr, n = (C.c_size_t * 1)(26), (C.c_size_t * 1)(11)
    config = abi.EnsembleConfig()
    config.count, config.nr, config.n = 1, nr, n
    config.drivers = C.pointer(driver)
    config.seed, config.fp32_bulk, config.dt_fraction = 3, bulk, 0.5
    e = lib.gcs_ensemble_create(C.byref(config))
    assert e, lib.gcs_last_error()
    alone = lib.gcs_context_create_wind(26, 11, 3, C.byref(driver))
    assert alone
    try:
        if bulk:
            assert lib.gcs_context_set_precision(alone, 1) == 0
        o, t = abi.AdvanceOptions(), abi.TimestepOptions()
        lib.gcs_case_options(2, C.byref(o), C.byref(t))
        bad = C.c_int()
        assert lib.gcs_ensemble_advance(e, 4) == 0
        assert lib.gcs_ensemble_sync(e, C.byref(bad)) == 0
        assert lib.gcs_context_run(alone, C.byref(o), C.byref(t), 0.5, 4, 1) == 0
        assert lib.gcs_context_sync(alone) == 0
        a, b = HostStorage([26, 11, 11], 4), HostStorage([26, 11, 11], 4)
        assert lib.gcs_context_download_state(lib.gcs_ensemble_run_context(e, 0),
                                              a.storage, 0) == 0
        assert lib.gcs_context_download_state(alone, b.storage, 0) == 0
        for f in range(6):
            x, y = a.arrays(f), b.arrays(f)
            for name in x:
                np.testing.assert_array_equal(x[name], y[name], err_msg=name)
    finally:
        lib.gcs_context_destroy(alone)
        lib.gcs_ensemble_destroy(e)


@pytest.mark.parametrize("nr,n,pinned", [(9, 9, False), (13, 10, True), (31, 17, False)])
def test_state_round_trip(lib, nr, n, pinned):
    """Random state arrays, uploaded and downloaded, come back bit for bit."""
    ctx = lib.gcs_context_create_case(1, nr, n, 1)
    assert ctx, lib.gcs_last_error()
    try:
        a = HostStorage([nr, n, n], 4, pinned=pinned, scratch=False)
        b = HostStorage([nr, n, n], 4, pinned=pinned, scratch=False)
        rng = np.random.default_rng(nr)
        for q in a._keep:
            np.asarray(q)[:] = rng.standard_normal(len(q))
        assert lib.gcs_context_upload_state(ctx, a.storage) == 0
        assert lib.gcs_context_download_state(ctx, b.storage, 0) == 0
        for x, y in zip(a._keep, b._keep):
            np.testing.assert_array_equal(np.asarray(x), np.asarray(y))
    finally:
        lib.gcs_context_destroy(ctx)



@pytest.mark.parametrize("nr,n", [(9, 9), (26, 11)])
def test_member_transfer_buffer(lib, nr, n):
    """A run that shares a grid moves its state through a buffer of five
    doubles a node of one face, the arrays one by one where they fill it:
    random states come back bit for bit, and the ensemble grows by no more
    than those buffers, which its admission estimate leaves out."""
    driver = (abi.WindDriver * 3)(*[abi.WindDriver(7.0, -420.0, 9e4, -4.0)] * 3)
    nrs, ns = (C.c_size_t * 3)(nr, nr, nr), (C.c_size_t * 3)(n, n, n)
    config = abi.EnsembleConfig(3, nrs, ns, driver, 3, 0, 0, 0.5)
    e = lib.gcs_ensemble_create(C.byref(config))
    assert e, lib.gcs_last_error()
    try:
        before = lib.gcs_ensemble_device_bytes(e)
        rng = np.random.default_rng(n)
        for run in range(3):
            ctx = lib.gcs_ensemble_run_context(e, run)
            a = HostStorage([nr, n, n], 4, scratch=False)
            b = HostStorage([nr, n, n], 4, scratch=False)
            for q in a._keep:
                q[:] = rng.standard_normal(len(q))
            assert lib.gcs_context_upload_state(ctx, a.storage) == 0
            assert lib.gcs_context_download_state(ctx, b.storage, 0) == 0
            for x, y in zip(a._keep, b._keep):
                np.testing.assert_array_equal(x, y)
        grown = lib.gcs_ensemble_device_bytes(e) - before
        assert 0 < grown <= 2 * 40 * (nr + 9) * (n + 9) * (n + 9)
    finally:
        lib.gcs_ensemble_destroy(e)


def test_failed_transfer_waits(lib):
    """A transfer that meets an array it cannot copy (a null pointer, which
    the copy call refuses) returns -1 only after the copies queued before it:
    the page-locked arrays they fill are the caller's to free then."""
    import torch
    nr, n = 64, 64
    ctx = lib.gcs_context_create_case(0, nr, n, 1)
    assert ctx, lib.gcs_last_error()
    try:
        want = HostStorage([nr, n, n], 4, pinned=True, scratch=False)
        got = HostStorage([nr, n, n], 4, pinned=True, scratch=False)
        assert lib.gcs_context_download_state(ctx, want.storage, 0) == 0
        for q in got._keep:
            q.fill_(-1.0)
        last = C.cast(got.storage[5].old_face_flux[2], C.c_void_p).value
        got.storage[5].old_face_flux[2] = None
        rc = lib.gcs_context_download_state(ctx, got.storage, 0)
        at_return = got._keep[-2].clone()   # face_flux[2], queued just before
        torch.cuda.synchronize()
        got.storage[5].old_face_flux[2] = C.cast(last, C.POINTER(C.c_double))
        assert rc == -1
        np.testing.assert_array_equal(at_return.numpy(), want._keep[-2].numpy())
        # the context goes on
        assert lib.gcs_context_download_state(ctx, got.storage, 0) == 0
        for x, y in zip(want._keep, got._keep):
            np.testing.assert_array_equal(x.numpy(), y.numpy())
    finally:
        lib.gcs_context_destroy(ctx)


def test_stage_times_name_what_ran(lib):
    """Profiled steps: every stage of the step has one call a step and its own
    time; recover_cfl, whose work is the update kernel's, has none."""
    ctx = lib.gcs_context_create_case(2, 12, 9, 1)
    assert ctx, lib.gcs_last_error()
    try:
        o, t = abi.AdvanceOptions(), abi.TimestepOptions()
        lib.gcs_case_options(2, C.byref(o), C.byref(t))
        assert lib.gcs_context_set_profiling(ctx, 1) == 0
        assert lib.gcs_context_run(ctx, C.byref(o), C.byref(t), 0.5, 3, 0) == 0
        ms, calls = (C.c_double * 16)(), (C.c_longlong * 16)()
        count = lib.gcs_context_stage_times(ctx, ms, calls, 16)
        got = {lib.gcs_stage_name(q).decode(): (calls[q], ms[q]) for q in range(count)}
        idle = {"recover_cfl", "mi_coupling"}
        for name, (n, time) in got.items():
            assert n == (0 if name in idle else 3), got
            assert (time > 0.0) == (name not in idle), got
    finally:
        lib.gcs_context_destroy(ctx)


def test_large_light_speeds(lib):
    """The Boris correction at light speeds whose square overflows in FP32 or
    FP64 (it does nothing there): one step against the restatement to 1e-12,
    and one FP32-bulk step against the FP64 one to 1e-5 of the largest EMF, a
    few dozen FP32 roundings (an Alfven speed lost to the overflow is 4e-5
    off in FP32, 1e-4 in FP64)."""
    ref, gpu = oracle_cases.pair("wind", 12, 9, 5)
    dt = 0.4 * ref.local_timestep()
    ctx = lib.gcs_context_create(gpu.grid, gpu.active, gpu.ghost)
    assert ctx, lib.gcs_last_error()
    try:
        assert lib.gcs_context_upload_background(ctx, gpu.background) == 0
        for light_speed in (10.0, 1e20, 1e160):
            for case in (ref, gpu):
                o = case.options[0]
                for group in (o.stress, o.emf, o.update):
                    assert group.use_boris
                    group.light_speed = light_speed
            done = [HostStorage(list(gpu.active), gpu.ghost) for _ in range(2)]
            for bulk in (0, 1):
                assert lib.gcs_context_set_precision(ctx, bulk) == 0
                assert lib.gcs_context_upload_state(ctx, gpu.storage) == 0
                if bulk and light_speed > 3e38:
                    break   # not an FP32 number: test_options_outside_fp32
                assert lib.gcs_context_step(ctx, gpu.options, 0.0, dt) == 0
                assert lib.gcs_context_download_state(ctx, done[bulk].storage, 1) == 0
            ref.copy_from(gpu)
            assert ref.step(0.0, dt) == 0
            bad = {k: v for k, v in compare_state(done[0], ref).items() if not v[0] <= 1e-12}
            assert not bad, (light_speed, bad)
            if light_speed > 3e38:
                continue
            for f in range(6):
                for e in range(3):
                    x, y = (s.arrays(f)["edge_emf%d" % e] for s in done)
                    assert np.abs(x - y).max() <= 1e-5 * np.abs(x).max(), light_speed
    finally:
        lib.gcs_context_destroy(ctx)


@pytest.mark.parametrize("gamma,light_speed,stage", [
    (5.0 / 3.0, 10.0, 0),
    (1.0 + 1e-9, 10.0, 4),     # 1 in FP32
    (5.0 / 3.0, 1e39, 5),      # infinite in FP32
    (5.0 / 3.0, 1e-39, 5),     # below the smallest normal FP32 number
])
def test_options_outside_fp32(lib, gamma, light_speed, stage):
    """gamma and c that FP32 cannot hold fail a step with FP32 layers, with the
    flux sweep's stage codes."""
    ctx = lib.gcs_context_create_case(2, 12, 9, 1)
    assert ctx, lib.gcs_last_error()
    try:
        o, t = abi.AdvanceOptions(), abi.TimestepOptions()
        lib.gcs_case_options(2, C.byref(o), C.byref(t))
        o.stress.gamma = o.update.gamma = gamma
        for group in (o.stress, o.emf, o.update):
            group.light_speed = light_speed
        assert lib.gcs_context_set_precision(ctx, 1) == 0
        rc = lib.gcs_context_step(ctx, C.byref(o), 0.0, 1e-6)
        assert lib.gcs_context_failure(ctx, None, None, None, None, None) == stage
        assert rc == (0 if stage == 0 else -1)
    finally:
        lib.gcs_context_destroy(ctx)


def test_more_layers_than_a_grid_dimension(lib):
    """22,000 radial layers: three families of them are more than grid.y's
    65535 blocks of one layer.  The step runs, and the uniform state keeps its
    CFL step."""
    import torch
    if torch.cuda.mem_get_info()[0] < 90e9:
        pytest.skip("needs 75 GB of device memory")
    ctx = lib.gcs_context_create_case(0, 22000, 9, 1)
    assert ctx, lib.gcs_last_error()
    try:
        o, t = abi.AdvanceOptions(), abi.TimestepOptions()
        lib.gcs_case_options(0, C.byref(o), C.byref(t))
        before, after = C.c_double(), C.c_double()
        assert lib.gcs_context_timestep(ctx, C.byref(t), C.byref(before)) == 0
        assert lib.gcs_context_step(ctx, C.byref(o), 0.0, 0.4 * before.value) == 0
        assert lib.gcs_context_timestep(ctx, C.byref(t), C.byref(after)) == 0
        # fluxes of 1 over layers 2e-5 thick cancel to rounding: 1e5 x 1e-16 x
        # a few dozen operations a step
        assert abs(after.value / before.value - 1.0) <= 1e-9
    finally:
        lib.gcs_context_destroy(ctx)
