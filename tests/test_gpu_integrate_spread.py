"""Integrate by four lanes per body (float64 batches of up to 8192 body rows):
the oracle's bits either side of the limit, with bodies that fall asleep or are
asleep, unnormalised and degenerate quaternions, and infinite masses."""
import numpy as np
import pytest

from cubez_gb300 import scenes
from oracle.oracle import FP64 as ORC_FP64
from oracle.oracle import OracleBatch

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0
FIELDS = ("position", "orientation", "velocity", "rotation", "motion", "is_awake", "inverse_inertia_world",
          "last_frame_acceleration")


@pytest.mark.parametrize("worlds,bodies", [(1, 1), (1, 7), (3, 33), (256, 32), (257, 32), (40, 64)])
def test_integrate_bit_exact(worlds, bodies, cuda_lib):
    from cubez_gb300.batch import WorldBatch
    scene = scenes.precision(num_worlds=worlds, bodies=bodies, seed=21)
    rng = np.random.default_rng(worlds + bodies)
    n = scene.num_bodies
    scene.can_sleep[:] = rng.random(n) < 0.6
    scene.is_awake[:] = rng.random(n) < 0.8
    scene.motion[:] = rng.uniform(0.0, 3.2, n)
    slow = rng.random(n) < 0.4
    scene.velocity[slow] *= 1e-3
    scene.rotation[slow] *= 1e-3
    scene.acceleration[rng.random(n) < 0.3] = 0.0
    scene.inverse_mass[rng.random(n) < 0.2] = 0.0
    scene.rotation[rng.random(n) < 0.3] *= 40.0
    scene.orientation[rng.random(n) < 0.2] *= 1.7
    scene.orientation[rng.random(n) < 0.05] = 0.0
    scene.linear_damping[:] = rng.choice([0.95, 1.0, 0.3], n)
    gpu = WorldBatch.from_scene(scene, form=0)
    ref = OracleBatch(scene, form=ORC_FP64)
    for _ in range(6):
        gpu.integrate(DT)
        ref.integrate(DT)
        g, r = gpu.download(FIELDS), ref.bodies()
        for k in FIELDS:
            if k in r:
                assert np.array_equal(g[k], r[k], equal_nan=g[k].dtype == np.float64), k
    assert np.array_equal(np.signbit(g["velocity"]), np.signbit(r["velocity"]))
