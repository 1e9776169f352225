"""The neighbour-list build against a plain search: particle counts around
the warp and tile edges, with and without boundary particles, particles with
equal keys, and particles with more neighbours than the build holds at once."""
import numpy as np
import pytest

from unifiedparticleframeworkcuda_b200 import FROZEN, LIQUID, UpfError, scenes

pytestmark = pytest.mark.gpu


def keys_of(p, x):
    """Morton keys in single precision (ZIndex::CalcIndex)."""
    c = np.array(p.scales[:], np.float32) * (x - np.array(p.zindex_origin[:], np.float32))
    c = np.clip(c, 0, 1023).astype(np.int64)
    key = np.zeros(len(x), np.int64)
    for b in range(10):
        for a in range(3):
            key |= ((c[:, a] >> b) & 1) << (3 * b + a)
    return key


def search(p, pos, typ):
    """{id: neighbour ids in list order}: everything nearer than h in float,
    by key, the dynamic particles before the boundary's at equal keys."""
    x = np.ascontiguousarray(pos[:, :3], np.float32)
    order = np.lexsort((np.arange(len(x)), typ == FROZEN, keys_of(p, x)))
    xs, h = x[order], np.float32(p.support_radius)
    out = {}
    for i in np.nonzero(typ != FROZEN)[0]:
        d = x[i] - xs
        r = np.sqrt((d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2])
        near = order[r < h]
        out[int(i)] = near[near != i]
    return out


def built(upf, p, pos, typ, **shape):
    s = upf.ParticleSystem(p, capacity=len(pos), derive=False)
    s.set_particles(pos, np.zeros_like(pos), typ)
    cfg = s.launch_config()
    for k, v in shape.items():
        setattr(cfg, k, v)
    s.set_launch_config(cfg)
    s.phase("sort")
    s.phase("neighbors")
    s.synchronize()
    counts, lists = s.neighbors()
    ids = s.sorted_keys()[1]
    s.close()
    return counts, lists, ids


def cloud(n, n_wall, seed, clump=0, gap=0.006):
    """n liquid and n_wall boundary particles in a box a few supports wide,
    `clump` of the liquid within a tenth of a support; some share a place."""
    p = scenes.small_pcisph().params
    p.max_neighbors = 512
    u = scenes.uniform(seed, 3 * (n + n_wall)).reshape(-1, 3)
    side = gap * (n + n_wall) ** (1 / 3) + 0.02
    pos = np.zeros((n + n_wall, 4), np.float32)
    pos[:, :3] = 0.03 + side * u
    pos[:clump, :3] = 0.05 + 0.002 * u[:clump]
    if n > 4:
        pos[n // 2, :3] = pos[0, :3]
    if n_wall > 4:
        pos[n + 1, :3] = pos[0, :3]
    typ = np.full(n + n_wall, LIQUID, np.int32)
    typ[n:] = FROZEN
    return p, pos, typ


@pytest.mark.parametrize("n,n_wall,clump", [(1, 0, 0), (1, 1, 0), (31, 0, 0), (33, 40, 0), (129, 1, 0), (700, 0, 300),
                                            (513, 600, 400), (3001, 997, 0)])
def test_lists_equal_a_plain_search(upf_lib, n, n_wall, clump):
    p, pos, typ = cloud(n, n_wall, seed=n, clump=clump)
    p = upf_lib.derive_params(p)
    want = search(p, pos, typ)
    for shape in ({}, {"nlist_threads": 64, "nlist_mode": 1}):
        counts, lists, ids = built(upf_lib, p, pos, typ, **shape)
        for c, row, i in zip(counts, lists, ids):
            assert np.array_equal(row[:c], want[int(i)]), (shape, int(i))


@pytest.mark.parametrize("n", [16384, 65536 + 17, 524288 + 5])
def test_particles_a_warp_do_not_change_the_lists(upf_lib, n):
    """The counts at which a warp takes more particles: both modes agree."""
    p, pos, typ = cloud(n, 1000, seed=3, gap=0.009)
    p.max_neighbors = 128
    p = upf_lib.derive_params(p)
    a = built(upf_lib, p, pos, typ)
    b = built(upf_lib, p, pos, typ, nlist_mode=1, nlist_threads=128)
    for u, v in zip(a, b):
        assert np.array_equal(u, v)


@pytest.mark.parametrize("n", [29999, 30000])
def test_counts_at_which_a_warp_takes_more(upf_lib, n):
    """Likewise on both sides of the count where it takes 16."""
    test_particles_a_warp_do_not_change_the_lists(upf_lib, n)


def test_more_neighbours_than_the_list_holds_is_an_error(upf_lib):
    p, pos, typ = cloud(700, 0, seed=9, clump=300)
    p.max_neighbors = 128
    with pytest.raises(UpfError) as e:
        built(upf_lib, upf_lib.derive_params(p), pos, typ)
    assert e.value.status == 4  # UPF_ERR_NEIGHBOR_OVERFLOW
