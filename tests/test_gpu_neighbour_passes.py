"""The list-based neighbour passes at the list lengths where they can go
wrong: bit for bit the pass that walks the cells (exact arithmetic) and the
shared-memory gather pipeline (fast arithmetic), which share no list walk with
them."""
import functools

import numpy as np
import pytest

import sph_gb300 as S
from helpers import REF, height_unit

pytestmark = pytest.mark.gpu

# particles of a cluster = in-range neighbours of each of them, itself included;
# around the pairs, quads and windows of 16 of the walks and the list's 192
SIZES = [1, 2, 3, 4, 5, 7, 8, 9, 12, 13, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 191, 192, 193, 200]
# particles of a second scene in the system: with 0 both passes take a group of
# lanes per particle, with 8,000 the fast force pass takes one lane, with 14,000
# the fast density pass too, with 20,000 all do
FILL = [0, 8000, 14000, 20000]
CELLS, GATHER = 0, 426232  # variants: cell walk; TMA gather pipeline


def clusters(rng, sizes, box=0.9, radius=0.006):
    """Clusters of the given sizes, 0.1 or more apart (h is 0.0457)."""
    centres = np.stack(np.meshgrid(*[np.arange(-box + 0.05, box, 0.11)] * 3, indexing="ij"), -1).reshape(-1, 3)
    centres = centres[rng.permutation(len(centres))[: len(sizes)]]
    pos = np.concatenate([c + rng.uniform(-radius, radius, (k, 3)) for c, k in zip(centres, sizes)])
    return pos[rng.permutation(len(pos))].astype(np.float32)


def case(name):
    rng = np.random.default_rng(41)
    pos = clusters(rng, SIZES)
    vel = rng.normal(0.0, 0.3, pos.shape).astype(np.float32)
    if name == "coincident":
        pos[5], pos[6], pos[7] = pos[4], pos[4], pos[8]
        vel[6] = vel[4]
        k = rng.permutation(np.arange(100, len(pos)))[:600]  # and pairs nearer than 1e-4
        pos[k[:300]] = pos[k[300:]] + rng.uniform(-5e-5, 5e-5, (300, 3))
    elif name == "infinite":
        vel[3, 1] = np.inf
        vel[10, 2] = -np.inf
        vel[11, 0] = np.nan
    return pos, vel


@functools.lru_cache(maxsize=None)
def records(name, cell_mult, variant, fill, record=True, tile=256):
    """Records after two steps of the clusters, beside `fill` other particles."""
    pos, vel = case(name)
    with S.System(particle_capacity=len(pos) + fill, variant=variant, tile=tile) as sysm:
        prm = dict(REF, box_len=0.9, cell_mult=cell_mult, flags=S.SPH_FLAG_RECORD if record else 0)
        sc = sysm.scene(S.default_params(**prm), capacity=len(pos))
        sc.set_particles(pos, vel)
        if fill:
            other = sysm.scene(S.default_params(**dict(prm, flags=0)), capacity=fill)
            other.set_particles(np.random.default_rng(1).uniform(-0.8, 0.8, (fill, 3)))
        sysm.step(2)
        return sc.get_records()


@pytest.mark.parametrize("cell_mult", [1.0, 0.5, 0.3])
@pytest.mark.parametrize("fill", FILL)
@pytest.mark.parametrize("name", ["plain", "coincident", "infinite"])
def test_list_lengths_bit_exact(name, fill, cell_mult):
    for reference, forms in ((CELLS, (88, 216)), (GATHER, (164088, 163960))):
        want = records(name, cell_mult, reference, FILL[-1])
        for v in forms:
            got = records(name, cell_mult, v, fill)
            assert np.array_equal(got[0], want[0], equal_nan=True), (reference, v)
            assert np.array_equal(got[1], want[1]), (reference, v)
        got = records(name, cell_mult, forms[0], fill, record=False, tile=128)
        assert np.array_equal(got[0][:, :6], want[0][:, :6], equal_nan=True), reference


def ordered(sizes, cell_mult, fill):
    """Records after two ordered steps of clusters, beside `fill` other particles."""
    rng = np.random.default_rng(7)
    pos = clusters(rng, sizes)
    vel = rng.normal(0.0, 0.3, pos.shape).astype(np.float32)
    pos[5], vel[3, 0] = pos[4], np.inf
    with S.System(particle_capacity=len(pos) + fill) as sysm:
        flags = S.SPH_FLAG_RECORD | S.SPH_FLAG_ORDERED
        prm = dict(REF, box_len=0.9, cell_mult=cell_mult)
        sc = sysm.scene(S.default_params(**prm, flags=flags), capacity=len(pos))
        sc.set_particles(pos, vel)
        if fill:
            sysm.scene(S.default_params(**prm)).set_particles(np.random.default_rng(1).uniform(-0.8, 0.8, (fill, 3)))
        sysm.step(2)
        return sc.get_records()


@pytest.mark.parametrize("cell_mult", [1.0, 0.5, 0.3])
def test_ordered_lists_bit_exact(cell_mult):
    """A warp per particle (few particles) against one lane per particle; more
    in-range neighbours than the ordered lists hold (128) are an error in both."""
    sizes = [k for k in SIZES if k <= 128] + [95, 96, 97]
    a, b = ordered(sizes, cell_mult, 0), ordered(sizes, cell_mult, 40000)
    assert np.array_equal(a[0], b[0], equal_nan=True) and np.array_equal(a[1], b[1])
    for fill in (0, 40000):
        with pytest.raises(S.SphError):
            ordered([129, 3], cell_mult, fill)


@pytest.mark.parametrize("cell_mult", [1.0, 0.25])
@pytest.mark.parametrize("n", [1, 33, 1023, 1024, 1025, 4095, 4096, 4097])
def test_one_block_sort(n, cell_mult):
    """The one-block sort of small scenes gives the keys, the stable order and
    the state after two steps of the sort over the whole system (taken when
    another scene is larger); grids of 1,000 to 60,000 keys."""
    rng = np.random.default_rng(n)
    pos = rng.uniform(-0.19, 0.19, (n, 3)).astype(np.float32)
    pos[: n // 7] = pos[0]  # a full cell
    vel = rng.normal(0.0, 0.3, pos.shape).astype(np.float32)
    out = []
    for fill in (0, 5000):
        with S.System(particle_capacity=n + fill) as sysm:
            prm = dict(REF, cell_mult=cell_mult)
            sc = sysm.scene(S.default_params(**prm, flags=S.SPH_FLAG_RECORD), capacity=n)
            sc.set_particles(pos, vel)
            if fill:
                sysm.scene(S.default_params(**prm)).set_particles(rng.uniform(-0.19, 0.19, (fill, 3)))
            sort = sc.debug_sort()
            sysm.step(2)
            out.append((*sort, *sc.get_records(), sc.debug_sort()[1]))
    for a, b in zip(*out):
        assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f")


@pytest.mark.parametrize("tile", [128, 256])
@pytest.mark.parametrize("shape", [(2, 2), (16, 8), (43, 3), (32, 28), (32, 32), (35, 33), (64, 65)])
def test_terrain_snapshot_of_every_tile(shape, tile):
    """The height snapshot is base + delta * unit at every vertex when the
    vertices are one tile or less, one more than a tile, and fill, underfill
    and overrun a block of several tiles."""
    rng = np.random.default_rng(5)
    base = rng.uniform(0.0, 0.1, shape[::-1]).astype(np.float32)
    pos = np.stack(np.meshgrid(*[np.linspace(-0.18, 0.18, 40)] * 2), -1).reshape(-1, 2)
    pos = np.insert(pos, 1, -0.15, axis=1).astype(np.float32)
    prm = dict(REF, dt=1e-3, erosion=1, k_capacity=0.05, erosion_layer=0.2)
    with S.System(tile=tile) as sysm:
        sc = sysm.scene(S.default_params(**prm), capacity=len(pos), terrain=shape)
        sc.set_terrain(base)
        sc.set_particles(pos, rng.normal(0.0, 1.0, pos.shape).astype(np.float32))
        sysm.step(3)
        h, delta = sc.get_terrain()
        assert sc.diag()["total_units"] == 0
    assert np.count_nonzero(delta) > delta.size // 8
    assert np.array_equal(h, base + delta.astype(np.float32) * height_unit(prm, shape))
