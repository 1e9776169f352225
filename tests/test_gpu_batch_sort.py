"""A batch's sort, one cluster a scene up to 65,536 particles and the general
sort where a scene is longer: every scene as when it is stepped alone, at both
sides of the rounds a cluster takes (4,096 particles each), bit for bit."""
import numpy as np
import pytest

from unifiedparticleframeworkcuda_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [(1,), (255, 256, 257), (4095, 4096, 4097, 1), (8192, 8193, 300), (40000, 12289, 24577),
                                    (65535, 61441), (65536, 7), (65537, 500), (70000, 65536, 3)])
def test_scenes_as_if_alone(upf_lib, counts):
    scs = [scenes.batch_scene(n, (0.8, 0.9 + 0.1 * k, 0.7), seed=3 + k, stream=k + 1) for k, n in enumerate(counts)]
    b = upf_lib.ParticleBatch.from_scenes(scs)
    b.step(2)
    got = [b.particles(k) for k in range(len(scs))]
    b.close()
    for sc, g in zip(scs, got):
        p = upf_lib.derive_params(sc.params)
        with upf_lib.ParticleSystem(p, capacity=sc.n, derive=False) as s:
            s.set_particles(sc.pos, sc.vel, sc.type)
            s.step(2)
            want = s.particles()
        for k in ("id", "pos", "vel", "density", "pressure"):
            assert np.array_equal(want[k], g[k]), (sc.n, k)
