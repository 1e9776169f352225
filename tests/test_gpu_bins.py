"""The density passes' table bin at squared distances too small for a normal
float."""
import ctypes as C

import numpy as np
import pytest

from unifiedparticleframeworkcuda_b200 import LIQUID, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [0.02, 0.04])
def test_subnormal_squared_distances_take_the_first_bin(upf_lib, h):
    p = upf_lib.default_params()
    p.support_radius = h
    tiny = np.float32(2.0 ** -149)
    r2 = np.array([tiny, 3 * tiny, 2.0 ** -140, 2.0 ** -127, np.nextafter(np.float32(2.0 ** -126), np.float32(0)),
                   2.0 ** -126, 0.0], np.float32)
    assert (r2[:5] > 0).all() and (r2[:5] < np.finfo(np.float32).tiny).all()
    out = np.full(r2.size, -1, np.int32)
    rc = upf_lib.lib().upf_selftest_support_bins(0, C.byref(p), r2.ctypes.data_as(C.POINTER(C.c_float)), r2.size,
                                                 out.ctypes.data_as(C.POINTER(C.c_int32)))
    assert rc == 0, upf_lib.lib().upf_last_error()
    assert not out.any(), out


# one launch for the whole loop, the TMA ring, direct loads, staged neighbourhoods
@pytest.mark.parametrize("shape", [None, (0, 128, 4), (1, 256, 4), (2, 256, 4)])
def test_particles_closer_than_the_root_of_the_smallest_normal_float(upf_lib, shape):
    """Two particles 1e-20 apart at the origin of coordinates see one another
    at full weight: twice the density of one alone."""
    sc = scenes.small_pcisph()
    sc.params.flags = 0
    sc.params.gravity = 0.0
    for f in ("collision_min", "container_min"):
        getattr(sc.params, f)[:] = (-0.3, -0.3, -0.3)
    sc.params.zindex_origin[:] = (-0.5, -0.5, -0.5)
    p = upf_lib.derive_params(sc.params)
    pos = np.zeros((2, 4), np.float32)
    pos[0, 0] = 1e-20
    densities = []
    for n in (1, 2):
        with upf_lib.ParticleSystem(p, capacity=2, derive=False) as s:
            s.set_particles(pos[:n], np.zeros((n, 4), np.float32), np.full(n, LIQUID, np.int32))
            if shape:
                c = s.launch_config()
                c.density_mode, c.density_threads, c.density_rows = shape
                c.pforce_mode, c.pforce_threads, c.pforce_rows = shape
                s.set_launch_config(c)
            s.step(1)
            s.synchronize()
            densities.append(s.step_fields()["predicted_density"])
    assert np.array_equal(densities[1], np.full(2, 2 * densities[0][0], np.float32))
