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
