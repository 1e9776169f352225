"""Which launches a step's predict-correct loop takes: the library's choice
while nothing is set, the caller's shapes from the first that is set, whatever
they are and whatever was set before, and the library's again after tuning."""
import ctypes as C

import numpy as np
import pytest

from unifiedparticleframeworkcuda_b200 import UpfLaunchConfig, scenes

pytestmark = pytest.mark.gpu

PASSES, ONE_LAUNCH, EITHER = 0, 1, 2


def route(upf, handle):
    r = C.c_int32(-1)
    batch = isinstance(handle, upf.ParticleBatch)
    f = upf.lib().upf_test_batch_loop_route if batch else upf.lib().upf_test_loop_route
    upf.check(f(handle.handle, C.byref(r)), "loop_route")
    return r.value


def loop_of(cfg):
    return (cfg.density_mode, cfg.density_threads, cfg.density_rows, cfg.pforce_mode, cfg.pforce_threads,
            cfg.pforce_rows)


def with_loop(cfg, loop):
    c = UpfLaunchConfig.from_buffer_copy(cfg)
    (c.density_mode, c.density_threads, c.density_rows, c.pforce_mode, c.pforce_threads, c.pforce_rows) = loop
    return c


def system(upf, sc):
    s = upf.ParticleSystem(upf.derive_params(sc.params), capacity=sc.n, derive=False)
    s.set_particles(sc.pos, sc.vel, sc.type)
    return s


OTHER = (0, 128, 4, 0, 128, 4)


@pytest.mark.parametrize("first", [None, OTHER])
def test_small_system(upf_lib, first):
    with system(upf_lib, scenes.small_pcisph()) as s:
        assert route(upf_lib, s) == ONE_LAUNCH
        stored = s.launch_config()
        if first:
            s.set_launch_config(with_loop(stored, first))
            assert route(upf_lib, s) == PASSES and loop_of(s.launch_config()) == first
        # the shapes that were stored from the beginning are a choice as well
        s.set_launch_config(stored)
        assert route(upf_lib, s) == PASSES and loop_of(s.launch_config()) == loop_of(stored)
        s.step(1)
        s.autotune(1)
        assert route(upf_lib, s) == ONE_LAUNCH
        s.step(1)
        s.synchronize()


def test_large_system_reports_and_honours_its_shapes(upf_lib):
    s = 0.01
    nx, ny, nz = 60, 54, 48
    sc = scenes.pcisph_dam(nx, ny, nz, seed=3, box=(s * (nx + 8), s * (ny + 4), s * (nz + 6)), spacing=s)
    with system(upf_lib, scenes.small_pcisph()) as small:
        stored = loop_of(small.launch_config())
    staged = (2, 256, 4, 2, 256, 4)
    with system(upf_lib, sc) as big:
        assert loop_of(big.launch_config()) == staged  # what its untuned steps run
        for loop in (stored, OTHER, stored, staged):
            big.set_launch_config(with_loop(big.launch_config(), loop))
            assert loop_of(big.launch_config()) == loop
            assert route(upf_lib, big) == PASSES
            big.step(1)
            big.synchronize()
        tuned = big.autotune(1)
        assert loop_of(big.launch_config()) == loop_of(tuned)


def test_batch(upf_lib):
    scs = scenes.batch_scenes(num=3, seed=13, counts=(2048, 4096))
    with upf_lib.ParticleBatch.from_scenes(scs) as b:
        assert route(upf_lib, b) == ONE_LAUNCH
        stored = b.launch_config()
        b.set_launch_config(stored)
        assert route(upf_lib, b) == PASSES
        b.step(1)
        b.autotune(1)
        assert route(upf_lib, b) == ONE_LAUNCH
        b.set_launch_config(with_loop(stored, OTHER))
        assert route(upf_lib, b) == PASSES
        b.autotune(1)
        assert route(upf_lib, b) == ONE_LAUNCH
        b.step(1)
        b.synchronize()


def end_state(handle, scenes_):
    got = [handle.particles(k) for k in range(scenes_)] if scenes_ else [handle.particles()]
    st = handle.stats()
    return got, [(s.iterations, s.total_iterations, s.max_predicted_density) for s in (st if scenes_ else [st])]


def same(a, b):
    assert a[1] == b[1]
    for u, v in zip(a[0], b[0]):
        for k in u:
            assert np.array_equal(u[k], v[k]), k


# what a step does beside other loops: its passes, for as long as they are
# there, and one launch again after them; at default and at tuned shapes
@pytest.mark.parametrize("loop", [None, (2, 256, 4, 2, 256, 8), (1, 256, 4, 0, 128, 4)])
def test_a_system_beside_others(upf_lib, loop):
    sc = scenes.pcisph_dam(20, 18, 16, seed=6, box=(0.3, 0.25, 0.25))
    with system(upf_lib, sc) as s, system(upf_lib, sc) as t:
        for _ in range(5):
            s.step(1)
        if loop:
            upf_lib.check(upf_lib.lib().upf_test_tuned_loop(t.handle, C.byref(with_loop(t.launch_config(), loop))),
                          "upf_test_tuned_loop")
        for meet in (False, True, True, False, False):
            if meet:
                upf_lib.check(upf_lib.lib().upf_test_meet_others(t.handle), "upf_test_meet_others")
            t.step(1)
        assert route(upf_lib, t) == EITHER and route(upf_lib, s) == ONE_LAUNCH
        same(end_state(t, 0), end_state(s, 0))


def test_a_batch_beside_others(upf_lib):
    scs = scenes.batch_scenes(num=4, seed=13, counts=(2048, 8192))
    with upf_lib.ParticleBatch.from_scenes(scs) as a, upf_lib.ParticleBatch.from_scenes(scs) as b:
        a.step(4)
        for meet in (True, True, False, False):
            if meet:
                upf_lib.check(upf_lib.lib().upf_test_batch_meet_others(b.handle), "upf_test_batch_meet_others")
            b.step(1)
        assert route(upf_lib, b) == EITHER and route(upf_lib, a) == ONE_LAUNCH
        same(end_state(b, 4), end_state(a, 4))


def test_a_call_of_many_steps(upf_lib):
    """As many calls of one step, for a system and a batch; then short calls."""
    sc = scenes.pcisph_dam(20, 18, 16, seed=6, box=(0.3, 0.25, 0.25))
    with system(upf_lib, sc) as s, system(upf_lib, sc) as t:
        for _ in range(19):
            s.step(1)
        t.step(17)
        assert route(upf_lib, t) == EITHER and route(upf_lib, s) == ONE_LAUNCH
        t.step(2)
        same(end_state(t, 0), end_state(s, 0))
    scs = scenes.batch_scenes(num=3, seed=13, counts=(2048, 4096))
    with upf_lib.ParticleBatch.from_scenes(scs) as a, upf_lib.ParticleBatch.from_scenes(scs) as b:
        for _ in range(17):
            a.step(1)
        b.step(16)
        b.step(1)
        assert route(upf_lib, b) == EITHER
        same(end_state(b, 3), end_state(a, 3))


def test_the_smallest_system_does_not_yield(upf_lib):
    with system(upf_lib, scenes.small_pcisph()) as s:
        upf_lib.check(upf_lib.lib().upf_test_meet_others(s.handle), "upf_test_meet_others")
        s.step(2)
        s.synchronize()
        assert route(upf_lib, s) == ONE_LAUNCH


def test_many_systems_at_once(upf_lib):
    """Six systems on streams of their own, stepped without waiting: each as
    if alone."""
    scs = [scenes.pcisph_dam(20 + k, 18, 17, seed=k, box=(0.35, 0.25, 0.25)) for k in range(6)]
    want = []
    for sc in scs:
        with system(upf_lib, sc) as s:
            s.step(8)
            want.append(end_state(s, 0))
    sys_ = [system(upf_lib, sc) for sc in scs]
    for _ in range(4):
        for s in sys_:
            s.step(1)
    for s in sys_:
        s.synchronize()
    for _ in range(4):
        for s in sys_:
            s.step(1)
    for s, w in zip(sys_, want):
        same(end_state(s, 0), w)
        s.close()
