"""The predict-correct loop in one launch against its passes as launches of
their own: every lane count and both list forms (held in shared memory, and
longer than what is held), systems and batches, bit for bit."""
import numpy as np
import pytest

from unifiedparticleframeworkcuda_b200 import FLAG_ADHESION, scenes

pytestmark = pytest.mark.gpu


def passes(handle):
    """Other loop shapes than the default ones: the passes as launches."""
    cfg = handle.launch_config()
    cfg.density_threads, cfg.density_rows = 128, 4
    cfg.pforce_threads, cfg.pforce_rows = 128, 4
    handle.set_launch_config(cfg)


def run_system(upf, sc, p, as_passes, steps):
    with upf.ParticleSystem(p, capacity=sc.n, derive=False) as s:
        s.set_particles(sc.pos, sc.vel, sc.type)
        if sc.num_bodies:
            s.set_rigid_bodies(sc.body, sc.num_bodies)
        if as_passes:
            passes(s)
        s.step(steps)
        st, g, f = s.stats(), s.particles(), s.step_fields()
        lag = s.lagged_state()
    f = {k: f[k][np.argsort(f["id"])] for k in ("pforce", "predicted_density")}
    return g, f, lag, (st.iterations, st.total_iterations, st.steps_at_max_loops, st.max_predicted_density,
                       list(st.iteration_max_density), st.max_step_density_error_percent)


# liquid particles (32, 16, 8, 4, 4, 2, 1 and 1 lanes a particle on a B200) and
# the support radius in spacings (2.7: 80 neighbours, more than a lane holds)
@pytest.mark.parametrize("block,h", [((5, 4, 3), 2.0), ((12, 12, 12), 2.0), ((12, 12, 12), 2.7), ((20, 17, 16), 2.0),
                                     ((25, 24, 23), 2.7), ((30, 28, 25), 2.0), ((37, 31, 25), 2.7),
                                     ((47, 39, 29), 2.7), ((50, 42, 31), 2.7), ((64, 43, 37), 2.0)])
def test_one_launch_equals_the_passes(upf_lib, block, h):
    nx, ny, nz = block
    s = 0.01
    sc = scenes.pcisph_dam(nx, ny, nz, seed=nx, box=(s * (nx + 8), s * (ny + 4), s * (nz + 6)), spacing=s)
    sc.params.support_radius = h * s
    sc.params.flags |= FLAG_ADHESION
    p = upf_lib.derive_params(sc.params)
    a = run_system(upf_lib, sc, p, False, 2)
    b = run_system(upf_lib, sc, p, True, 2)
    assert a[3] == b[3]
    for u, v in ((a[0], b[0]), (a[1], b[1])):
        for k in u:
            assert np.array_equal(u[k], v[k]), k
    assert np.array_equal(a[2], b[2])


def test_one_launch_with_bodies_and_grains(upf_lib):
    sc = scenes.small_coupling()
    p = upf_lib.derive_params(sc.params)
    a = run_system(upf_lib, sc, p, False, 5)
    b = run_system(upf_lib, sc, p, True, 5)
    assert a[3] == b[3]
    for k in a[0]:
        assert np.array_equal(a[0][k], b[0][k]), k


@pytest.mark.parametrize("counts", [(1, 700, 257), (2048, 300, 5000, 900), (9000, 40, 30000), (65536, 3000, 50000)])
def test_one_launch_over_a_batch(upf_lib, counts):
    """Scenes that end their loops after different numbers of iterations."""
    scs = [scenes.batch_scene(n, (0.6, 0.5 + 0.1 * k, 0.7), seed=5 + k, stream=k + 1) for k, n in enumerate(counts)]
    got = []
    for as_passes in (False, True):
        b = upf_lib.ParticleBatch.from_scenes(scs)
        if as_passes:
            passes(b)
        b.step(3)
        got.append(([b.particles(k) for k in range(len(scs))],
                    [(s.iterations, s.total_iterations, s.total_steps, s.max_predicted_density) for s in b.stats()]))
        b.close()
    assert got[0][1] == got[1][1]
    for u, v in zip(got[0][0], got[1][0]):
        for k in u:
            assert np.array_equal(u[k], v[k]), k


def test_systems_on_streams_of_their_own(upf_lib):
    """Three systems stepped at the same time, each on its own stream: every
    one as if alone."""
    scs = [scenes.pcisph_dam(20 + 9 * k, 20, 20, seed=k, box=(0.7, 0.3, 0.3)) for k in range(3)]
    ps = [upf_lib.derive_params(sc.params) for sc in scs]
    alone = [run_system(upf_lib, sc, p, False, 6) for sc, p in zip(scs, ps)]
    sys_ = [upf_lib.ParticleSystem(p, capacity=sc.n, derive=False) for sc, p in zip(scs, ps)]
    for s, sc in zip(sys_, scs):
        s.set_particles(sc.pos, sc.vel, sc.type)
    for _ in range(6):
        for s in sys_:
            s.step(1)
    for s, a in zip(sys_, alone):
        g = s.particles()
        for k in g:
            assert np.array_equal(g[k], a[0][k]), k
        s.close()
