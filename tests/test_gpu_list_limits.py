"""The list passes past their limits: more neighbours in range than the list
and the group passes' term buffer hold, and packed records that an HBM budget
takes back between steps."""
import numpy as np
import pytest

import sph_gb300 as S
from helpers import REF
from test_gpu_neighbour_passes import CELLS, FILL, GATHER, clusters

pytestmark = pytest.mark.gpu

SIZES = [223, 224, 225, 255, 256, 257, 300, 3, 1]  # around the 224 in range at which terms are first added


def records(variant, cell_mult, fill):
    rng = np.random.default_rng(19)
    pos = clusters(rng, SIZES)
    vel = rng.normal(0.0, 0.3, pos.shape).astype(np.float32)
    with S.System(particle_capacity=len(pos) + fill, variant=variant) as sysm:
        prm = dict(REF, box_len=0.9, cell_mult=cell_mult)
        sc = sysm.scene(S.default_params(**prm, flags=S.SPH_FLAG_RECORD), capacity=len(pos))
        sc.set_particles(pos, vel)
        if fill:
            other = sysm.scene(S.default_params(**prm), capacity=fill)
            other.set_particles(np.random.default_rng(1).uniform(-0.8, 0.8, (fill, 3)))
        sysm.step(2)
        return sc.get_records()


@pytest.mark.parametrize("cell_mult", [1.0, 0.3])
@pytest.mark.parametrize("fill", FILL)
@pytest.mark.parametrize("reference,variant", [(CELLS, 88), (GATHER, 163960)])
def test_long_lists_bit_exact(reference, variant, fill, cell_mult):
    want, got = records(reference, cell_mult, FILL[-1]), records(variant, cell_mult, fill)
    assert np.array_equal(got[0], want[0], equal_nan=True) and np.array_equal(got[1], want[1])


def run(variant, budget):
    """Two scenes in an arena of 65,536 particles; the second one's terrain
    grows to 1,500 x 1,500 between steps."""
    caps = (24576, 40960)
    rng = np.random.default_rng(2)
    out, mem = [], []
    with S.System(particle_capacity=caps[0], variant=variant, hbm_budget=budget) as sysm:
        prm = S.default_params(**dict(REF, box_len=0.4))
        scenes = [sysm.scene(prm, capacity=n, terrain=(64, 64)) for n in caps]
        for sc, n in zip(scenes, caps):
            sc.set_particles(rng.uniform(-0.35, 0.35, (n, 3)).astype(np.float32))
        sysm.step(2)
        mem.append(sysm.memory())
        scenes[1].set_terrain(np.zeros((1500, 1500), np.float32))
        mem.append(sysm.memory())
        sysm.step(2)
        mem.append(sysm.memory())
        for sc in scenes:
            st = sc.get_particles()
            out += [st["pos"], st["vel"], st["density"]]
    return out, mem


@pytest.mark.parametrize("variant", [88, 163960])
def test_budget_takes_the_records_back(variant):
    want, free = run(variant, 0)
    records = 32 * 65536
    budget = free[2] - records + 4096
    got, held = run(variant, budget)
    assert held[0] == free[0]  # they fit at first
    assert held[1] == free[1] - records and held[2] == free[2] - records <= budget
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
