"""A host radial boundary callback that sets the two sides of an active seam
face apart, against the restatement with the same callback."""
import ctypes as C

import pytest

from gamera_cube_b200 import abi
from oracle import oracle_cases
from tests.parity_util import compare_state

pytestmark = pytest.mark.gpu

RADIAL = C.CFUNCTYPE(C.c_int, C.POINTER(abi.Grid), C.POINTER(abi.Storage),
                     C.POINTER(C.c_size_t), C.c_size_t, C.c_double, C.c_double, C.c_void_p)


@pytest.fixture(scope="module")
def lib():
    import gamera_cube_b200
    return gamera_cube_b200.lib


@pytest.mark.parametrize("kind", ["wind", "shock"])
def test_callback_may_set_seam_sides_apart(lib, kind):
    """Phi of one side of every axis-1 and axis-2 seam face 1 % (and Phi_old
    2 %) off after the halo fills: the momentum update of the cells beside the
    seams takes each side's own Phi, the stored B the mean of the two."""
    ref, gpu = oracle_cases.pair(kind, 12, 9, 5)
    g, (nr, n) = ref.ghost, list(ref.active)[:2]

    @RADIAL
    def radial(_grid, storage, _active, _ghost, _time, _previous, _context):
        for f in (0, 3):
            a = abi.storage_arrays(storage[f])
            for name, by in (("face_flux", 1.01), ("old_face_flux", 1.02)):
                a[name + "1"][g:g + nr, g + n, g:g + n] *= by
                a[name + "2"][g:g + nr, g:g + n, g] *= by
        return 0

    address = C.cast(radial, C.c_void_p)
    plan = C.c_void_p()
    assert lib.gamera_cs_halo_plan_create(gpu.grid, gpu.active, gpu.ghost,
                                          C.byref(plan)) == 0, lib.gcs_last_error()
    try:
        dt = 0.4 * ref.local_timestep()
        for ratio in (0.0, 0.5):
            assert oracle_cases.lib().gcso_case_step_radial(ref.handle, ratio, dt, address,
                                                            None) == 0
            assert lib.gamera_cs_advance_six_with_background_planned(
                gpu.grid, gpu.storage, gpu.active, gpu.ghost, ratio, dt, gpu.options,
                gpu.background, plan, address, 0.0, 0.0, None) == 0
            bad = {k: v for k, v in compare_state(gpu, ref).items() if not v[0] <= 1e-12}
            assert not bad, bad
            gpu.copy_from(ref)
    finally:
        lib.gamera_cs_halo_plan_destroy(plan)
