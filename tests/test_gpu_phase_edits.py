"""Arrays that a caller may replace between the phases (upf_get_device_state):
what it writes is what the next phase reads."""
import ctypes as C

import numpy as np
import pytest
import torch

from unifiedparticleframeworkcuda_b200 import (FLAG_SURFACE_TENSION, FLAG_WALL_WEIGHT, FROZEN, RIGID, UpfDeviceState,
                                                scenes)

pytestmark = pytest.mark.gpu


class View:
    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "version": 3, "strides": None,
                                         "data": (C.cast(ptr, C.c_void_p).value, False)}


def arrays(upf, s):
    d = UpfDeviceState()
    upf.check(upf.lib().upf_get_device_state(s.handle, C.byref(d)), "upf_get_device_state")
    return {k: torch.as_tensor(View(getattr(d, k), (d.n, 4) if k.endswith("4") else (d.n,)), device="cuda")
            for k in ("sorted_pos4", "density", "pressure")}


# four lanes a particle and one
@pytest.mark.parametrize("side", [12, 41])
def test_wcsph_density_and_pressure_between_forces_and_integration(upf_lib, side):
    """Densities and pressures of a stiffer system with wall weights, written
    over those of a softer one without: the integration, which takes nothing
    else from either parameter, gives the stiffer system's state."""
    sc = scenes.wcsph_dam(side, seed=side, box=0.02 * (side + 10))
    sc.params.dt = 5e-4
    sc.type[np.arange(9) * 23] = RIGID
    soft, stiff = sc.params.copy(), sc.params.copy()
    soft.flags = FLAG_SURFACE_TENSION
    stiff.flags = FLAG_SURFACE_TENSION | FLAG_WALL_WEIGHT
    stiff.gas_constant *= 2

    def run(params, given=None):
        with upf_lib.ParticleSystem(upf_lib.derive_params(params), capacity=sc.n, derive=False) as s:
            s.set_particles(sc.pos, sc.vel, sc.type)
            for ph in ("sort", "neighbors", "forces"):
                s.phase(ph)
            s.synchronize()
            a = arrays(upf_lib, s)
            found = {k: a[k].clone() for k in ("density", "pressure")}
            for k in given or ():
                a[k].copy_(given[k])
            torch.cuda.synchronize()
            s.phase("integrate")
            s.synchronize()
            return s.particles(), found

    want, given = run(stiff)
    plain, _ = run(soft)
    got, _ = run(soft, given)
    assert not np.array_equal(plain["vel"], want["vel"])
    for k in want:
        assert np.array_equal(got[k], want[k]), k


@pytest.mark.parametrize("scene", ["small_pcisph", "small_wcsph"])
def test_positions_between_sort_and_lists(upf_lib, scene):
    """Sorted positions moved by the caller: the lists are those of the moved
    positions, with boundary particles in the scene."""
    sc = getattr(scenes, scene)()
    p = upf_lib.derive_params(sc.params)
    h = np.float32(p.support_radius)
    wall = np.flatnonzero(sc.type == FROZEN)
    with upf_lib.ParticleSystem(p, capacity=sc.n, derive=False) as s:
        s.set_particles(sc.pos, sc.vel, sc.type)
        s.phase("sort")
        s.synchronize()
        ids = s.sorted_keys()[1]
        a = arrays(upf_lib, s)["sorted_pos4"]
        # under half a grid unit to either side: within the margin of the cells
        shift = np.float32(0.05 * p.particle_spacing) * np.where(np.arange(len(ids)) % 2, 1, -1).astype(np.float32)
        a[:, 0] += torch.as_tensor(shift, device="cuda")
        torch.cuda.synchronize()
        x = sc.pos[:, :3].astype(np.float32).copy()
        x[ids] = a.cpu().numpy()[:, :3]
        s.phase("neighbors")
        s.synchronize()
        counts, lists = s.neighbors()
    every = np.concatenate([ids.astype(np.int64), wall])
    for k in range(0, len(ids), 7):
        i = int(ids[k])
        d = x[i] - x[every]
        r = np.sqrt((d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2])
        want = np.sort(every[(r < h) & (every != i)])
        assert np.array_equal(np.sort(lists[k, :counts[k]]).astype(np.int64), want), i
