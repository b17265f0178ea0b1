"""The list-based neighbour passes at the list lengths where they can go
wrong: bit for bit the pass that walks the cells (exact arithmetic) and the
shared-memory gather pipeline (fast arithmetic), which share no list walk with
them."""
import numpy as np
import pytest

import sph_gb300 as S
from helpers import REF, run

pytestmark = pytest.mark.gpu

# particles of a cluster = in-range neighbours of each of them, itself included;
# around the pairs, quads and rings of four of the walks and the list's 192
SIZES = [1, 2, 3, 4, 5, 7, 8, 9, 12, 13, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 191, 192, 193, 200]


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
    elif name == "infinite":
        vel[3, 1] = np.inf
        vel[10, 2] = -np.inf
        vel[11, 0] = np.nan
    return pos, vel


@pytest.mark.parametrize("cell_mult", [1.0, 0.5, 0.3])
@pytest.mark.parametrize("name", ["plain", "coincident", "infinite"])
def test_list_lengths_bit_exact(name, cell_mult):
    pos, vel = case(name)
    prm = dict(REF, box_len=0.9)
    for ref, forms in ((0, (88, 216)), (426232, (164088, 163960))):
        want = run(prm, pos, 2, vel=vel, cell_mult=cell_mult, variant=ref)[2]
        for v in forms:
            for record in (True, False):
                flags = S.SPH_FLAG_RECORD if record else 0
                got = run(prm, pos, 2, vel=vel, cell_mult=cell_mult, variant=v, flags=flags)[2]
                cols = slice(0, 27) if record else slice(0, 6)
                assert np.array_equal(got[0][:, cols], want[0][:, cols], equal_nan=True), (ref, v, record)
                if record:
                    assert np.array_equal(got[1], want[1]), (ref, v)
