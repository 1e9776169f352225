"""The WCSPH step's fused density and its force pass, at one and four lanes a
particle: against the oracle within the parity bar, and against the phase
entry points (density as a pass of its own) bit for bit."""
import numpy as np
import pytest

from test_gpu_parity import RTOL, _compare_step, make
from unifiedparticleframeworkcuda_b200 import (FLAG_SURFACE_TENSION, FLAG_WALL_WEIGHT, RIGID, scenes)

pytestmark = pytest.mark.gpu


# below and above the size at which a particle takes one lane; with and
# without the third term; some dynamic particles that are not liquid
@pytest.mark.parametrize("side,flags,rigid", [(5, 0, 0), (13, 0, 7), (13, FLAG_SURFACE_TENSION, 7),
                                              (41, FLAG_SURFACE_TENSION | FLAG_WALL_WEIGHT, 50), (41, 0, 0)])
def test_step_equals_phases_and_oracle(upf_lib, oracle_lib, side, flags, rigid):
    sc = scenes.wcsph_dam(side, seed=side, box=max(0.3, 0.02 * (side + 10)))
    sc.params.dt = 5e-4
    sc.params.flags = flags
    if rigid:
        sc.type[np.arange(rigid) * 23] = RIGID
    p, s, o = make(upf_lib, oracle_lib, sc)
    s.step(1)
    o.step()
    bad = {k: v for k, v in _compare_step(s, o, "wcsph").items() if not v[0]}
    assert not bad, "fields beyond %g relative: %s" % (RTOL, bad)
    o.close()
    s.step(2)
    with upf_lib.ParticleSystem(p, capacity=sc.n, derive=False) as t:
        t.set_particles(sc.pos, sc.vel, sc.type)
        for _ in range(3):
            for phase in ("sort", "neighbors", "forces", "integrate"):
                t.phase(phase)
        a, b = s.particles(), t.particles()
    s.close()
    for k in a:
        assert np.array_equal(a[k], b[k]), k


# the sizes nearest the line between four lanes and one
@pytest.mark.parametrize("side", [31, 32])
def test_step_equals_phases_and_oracle_at_the_line(upf_lib, oracle_lib, side):
    test_step_equals_phases_and_oracle(upf_lib, oracle_lib, side, FLAG_SURFACE_TENSION, 7)
