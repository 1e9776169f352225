"""The adjoint's step graphs: intervals that divide the trajectory or leave a
shorter last one, one or several loop iterations, and repeated calls with
other velocities and viscosities, all bit for bit the same trajectory and
gradient."""
import numpy as np
import pytest

from unifiedparticleframeworkcuda_b200 import scenes

pytestmark = pytest.mark.gpu

STEPS = 7


def gradient(upf, sc, interval, loops, calls, **kw):
    """(loss, gradient, viscosity gradient, final state) of the last of `calls`
    (velocity scale, viscosity) on one handle."""
    a = upf.Adjoint(sc.params, sc.pos, sc.vel, steps=STEPS, checkpoint_interval=interval, loop_iterations=loops,
                    target=(1.0, 1.0, 1.0), **kw)
    for scale, mu in calls:
        loss = a.forward(sc.vel * np.float32(scale), mu)
        g, gm = a.backward()
    out = loss, g, gm, a.state()
    a.close()
    return out


@pytest.mark.parametrize("n", [(5, 3, 3), (17, 16, 16), (40, 32, 33)])  # one warp; small and large CTAs
@pytest.mark.parametrize("loops", [1, 3])
def test_intervals_and_repeats_agree(upf_lib, n, loops):
    sc = scenes.adjoint_scene(*n, seed=sum(n))
    ref = gradient(upf_lib, sc, STEPS, loops, [(1.0, 0.7)])
    for interval in (1, 3):
        for calls in ([(1.0, 0.7)], [(0.3, 2.0), (1.0, 0.7)]):
            got = gradient(upf_lib, sc, interval, loops, calls)
            assert np.array_equal(got[1], ref[1])
            for u, v in zip(got[3], ref[3]):
                assert np.array_equal(u, v)
            # sums over blocks in double, in no fixed order
            assert got[0] == pytest.approx(ref[0], rel=1e-13)
            assert got[2] == pytest.approx(ref[2], rel=1e-11)


@pytest.mark.parametrize("interval", [2, STEPS])
def test_two_gradients_of_one_forward(upf_lib, interval):
    """A second backward after one forward gives the first one's gradient."""
    sc = scenes.adjoint_scene(9, 8, 7, seed=4)
    with upf_lib.Adjoint(sc.params, sc.pos, sc.vel, steps=STEPS, checkpoint_interval=interval, loop_iterations=3,
                         target=(1.0, 1.0, 1.0)) as a:
        a.forward(sc.vel, 0.7)
        g, gm = a.backward()
        assert np.abs(g).max() > 0
        for _ in range(2):
            g2, gm2 = a.backward()
            assert np.array_equal(g2, g)
            assert gm2 == pytest.approx(gm, rel=1e-11)  # a sum over blocks in double, in no fixed order
        x = a.state()
        a.forward(sc.vel, 0.7)
        g3, _ = a.backward()
        assert np.array_equal(g3, g)
        for u, v in zip(a.state(), x):
            assert np.array_equal(u, v)


def test_no_gradient_of_a_forward_that_failed(upf_lib):
    """A forward whose particles gather more neighbours than the lists hold
    leaves no trajectory to differentiate; the next good one does."""
    from unifiedparticleframeworkcuda_b200 import STATUS, UpfError
    sc = scenes.adjoint_scene(8, 8, 8, seed=4)
    inward = np.zeros_like(sc.vel)
    inward[:, :3] = (sc.pos[:, :3].mean(0) - sc.pos[:, :3]) / (2 * STEPS * sc.params.dt)
    p = upf_lib.derive_params(sc.params)

    def handle(max_neighbors):
        p.max_neighbors = max_neighbors
        return upf_lib.Adjoint(p, sc.pos, sc.vel, steps=STEPS, checkpoint_interval=3, loop_iterations=1,
                               target=(1.0, 1.0, 1.0), derive=False)

    def fails(a, vel):
        try:
            a.forward(vel, 0.7)
        except UpfError as e:
            assert STATUS[e.status] == "UPF_ERR_NEIGHBOR_OVERFLOW"
            return True
        return False

    # the fewest neighbours that the good trajectory gets by with
    room = 8
    while True:
        with handle(room) as a:
            if not fails(a, sc.vel):
                break
        room += 1
    with handle(room) as a:
        loss = a.forward(sc.vel, 0.7)
        g, _ = a.backward()
        assert fails(a, inward)
        for call in (a.backward, a.state):
            with pytest.raises(UpfError) as e:
                call()
            assert STATUS[e.value.status] == "UPF_ERR_STATE"
        assert a.forward(sc.vel, 0.7) == pytest.approx(loss, rel=1e-13)
        assert np.array_equal(a.backward()[0], g)
