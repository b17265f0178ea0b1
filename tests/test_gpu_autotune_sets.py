"""Variants that launch the same kernels are one candidate of the autotuner."""
import pytest

import sph_gb300 as S
import workloads as W

pytestmark = pytest.mark.gpu

EXACT, FAST = {28, 88, 120, 216, 32856, 32888}, {163928, 163960, 164088}


@pytest.mark.parametrize("flags", [0, S.SPH_FLAG_RECORD])
def test_variants_of_the_same_kernels_are_timed_once(flags):
    """They share one time, and the one picked asks for no memory that changes
    nothing (bit 128)."""
    with S.System(tile=256) as sysm:
        sysm.scene_from_request(W.base_params(1.0), dict(seed=5, particles=6000, terrain_side=64, steps=0))
        if flags:
            pos = W.lattice_block(8, 8, 8, W.SPACING, (-0.1, -0.1, -0.1))
            sysm.scene(S.default_params(**dict(W.PHYS, flags=flags))).set_particles(pos)
        sysm.step(5)
        tuned = sysm.autotune(2)
    for tile in (128, 256):
        for cm in (1.0, 0.5):
            ms = {v: t for ti, c, v, t in tuned["tried"] if (ti, c) == (tile, cm)}
            assert len(ms) == 14
            for same in (EXACT, FAST):
                assert len({ms[v] for v in same}) == 1
            assert len(set(ms.values())) >= 3  # other kernels are timed by themselves
    assert not tuned["variant"] & 128
