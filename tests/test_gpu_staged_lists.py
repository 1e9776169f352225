"""The staged loop passes take a list's entries in whole batches: what lies
past a list's end must not reach the sums, also where a list is full and its
capacity no multiple of a batch, or where a pressure is not finite. Each case bit for bit against passes that
stop at the list's end."""
import numpy as np
import pytest

from unifiedparticleframeworkcuda_b200 import LIQUID, scenes

pytestmark = pytest.mark.gpu

FIELDS = ("pos", "vel", "density", "pressure")


def loop_shape(s, mode, threads, rows):
    c = s.launch_config()
    c.density_mode, c.density_threads, c.density_rows = mode, threads, rows
    c.pforce_mode, c.pforce_threads, c.pforce_rows = mode, threads, rows
    s.set_launch_config(c)


def one_step(upf, p, pos, vel, typ, shape, seen=None):
    with upf.ParticleSystem(p, capacity=len(pos), derive=False) as s:
        s.set_particles(pos, vel, typ)
        if shape:
            loop_shape(s, *shape)
        # NaN wherever the list build writes nothing
        upf.check(upf.lib().upf_test_fill_list_values(s.handle, 0xff), "upf_test_fill_list_values")
        s.step(1)
        st, g = s.stats(), s.particles()
    o = np.argsort(g["id"], kind="stable")
    if seen is not None:
        seen.append(st.max_neighbor_count)
    return {k: g[k][o] for k in FIELDS}, st.iterations


# below and above the size from which untuned steps are staged (shape None)
@pytest.mark.parametrize("block,shapes", [((12, 12, 12), [(2, 256, 4), (2, 256, 8)]),
                                          ((60, 54, 48), [None, (2, 256, 4), (2, 256, 8)])])
def test_lists_filled_to_a_capacity_that_is_no_multiple_of_four(upf_lib, block, shapes):
    s = 0.01
    nx, ny, nz = block
    sc = scenes.pcisph_dam(nx, ny, nz, seed=3, box=(s * (nx + 8), s * (ny + 4), s * (nz + 6)), spacing=s)
    for h in (2.0, 2.05, 2.1, 2.15, 2.2):  # until the longest list is no whole number of batches
        sc.params.support_radius = h * s
        p = upf_lib.derive_params(sc.params)
        seen = []
        want = one_step(upf_lib, p, sc.pos, sc.vel, sc.type, (0, 128, 4), seen)
        if seen[0] % 4:
            break
    assert seen[0] % 4
    p.max_neighbors = seen[0]
    for shape in [(0, 128, 4), (1, 256, 4)] + shapes:
        got = one_step(upf_lib, p, sc.pos, sc.vel, sc.type, shape)
        assert got[1] == want[1], shape
        for k in FIELDS:
            assert np.array_equal(got[0][k], want[0][k]), (shape, k)


@pytest.mark.parametrize("rows", [4, 8])
def test_a_pressure_that_is_not_finite(upf_lib, rows):
    """Two particles whose correction pressure overflows: each is thrown
    against the walls by the infinite force of its one neighbour, and the
    batch's three other entries add nothing to it."""
    sc = scenes.small_pcisph()
    sc.params.flags = 0
    p = upf_lib.derive_params(sc.params)
    p.mass *= 4.0
    p.density_error_factor = 1e38
    mid = 0.5 * (np.array(p.collision_min[:]) + np.array(p.collision_max[:]))
    pos = np.zeros((2, 4), np.float32)
    pos[0, :3] = mid - 0.002
    pos[1, :3] = mid + 0.002
    vel, typ = np.zeros_like(pos), np.full(2, LIQUID, np.int32)
    want = one_step(upf_lib, p, pos, vel, typ, (0, 128, 4))
    assert np.isinf(want[0]["pressure"]).all() and np.isfinite(want[0]["pos"]).all()
    got = one_step(upf_lib, p, pos, vel, typ, (2, 256, rows))
    assert got[1] == want[1]
    for k in FIELDS:
        assert np.array_equal(got[0][k], want[0][k]), k
