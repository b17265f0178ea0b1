"""A particle without neighbours gets no pressure force whatever its pressure:
its pair with itself adds to the colour field alone, also where that pair's
pressure factor, which nothing uses, exceeds the range of a float."""
import numpy as np
import pytest

import sph_gb300 as S
from helpers import REF, FIELDS

pytestmark = pytest.mark.gpu

FILL = 20000  # particles of a second scene: enough for the passes over packed records


def records(variant, pressure_factor):
    """Records after one step of particles 0.11 apart (h is 0.0457) whose
    P / rho^2 is -pressure_factor."""
    h, mass, rho0 = REF["smoothing_radius"], 5e-5, REF["rest_density"]
    rho = mass * 315.0 / (64.0 * np.pi * h ** 3)  # a particle's own density
    prm = dict(REF, box_len=0.9, mass=mass, gas_stiffness=pressure_factor * rho * rho / (rho0 - rho))
    pos = np.stack(np.meshgrid(*[np.arange(-0.85, 0.86, 0.11)] * 3, indexing="ij"), -1).reshape(-1, 3)[::7]
    vel = np.random.default_rng(3).normal(0.0, 0.3, pos.shape).astype(np.float32)
    with S.System(particle_capacity=len(pos) + FILL, variant=variant) as sysm:
        sc = sysm.scene(S.default_params(**prm, flags=S.SPH_FLAG_RECORD), capacity=len(pos))
        sc.set_particles(pos.astype(np.float32), vel)
        other = sysm.scene(S.default_params(**dict(REF, box_len=0.9)), capacity=FILL)
        other.set_particles(np.random.default_rng(1).uniform(-0.8, 0.8, (FILL, 3)))
        sysm.step(1)
        return sc.get_records()


@pytest.mark.parametrize("pressure_factor", [1e20, 1e33, 2.4e38])
@pytest.mark.parametrize("reference,variant", [(0, 88), (0, 216), (426232, 163960), (426232, 164088)])
def test_large_pressure_alone_exerts_no_force(reference, variant, pressure_factor):
    want, got = records(reference, pressure_factor), records(variant, pressure_factor)
    assert np.isfinite(want[0][:, :26]).all() and (want[0][:, FIELDS["fpress"]] == 0).all()
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
