"""Host copies of the body state (cz_upload_bodies, cz_download_bodies): any
choice of fields gives what all of them give, for arrays copied by one thread
and by several, and damping factors that change from body to body or not."""
import numpy as np
import pytest

from cubez_gb300 import scenes
from oracle.oracle import FP32 as ORC_FP32
from oracle.oracle import FP64 as ORC_FP64
from oracle.oracle import OracleBatch

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0
FIELDS = ("position", "orientation", "velocity", "rotation", "acceleration", "inverse_inertia", "inverse_mass",
          "linear_damping", "angular_damping", "motion", "is_awake", "can_sleep", "shape", "half_size", "radius",
          "inverse_inertia_world", "last_frame_acceleration", "collider_offset")


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("worlds,bodies", [(1, 3), (40, 9), (1700, 30)])
def test_fields_chosen_at_will(form, worlds, bodies, cuda_lib):
    from cubez_gb300.batch import WorldBatch
    scene = scenes.offsets(num_worlds=worlds, bodies=bodies, seed=3)
    gpu = WorldBatch.from_scene(scene, form=form)
    gpu.step(2, DT)
    every = gpu.download(FIELDS)
    for k in ("shape", "can_sleep", "linear_damping", "angular_damping"):
        assert np.array_equal(every[k], getattr(scene, k)), k
    for pick in [(k,) for k in FIELDS] + [FIELDS[::2], FIELDS[1::3], ("motion", "position"), ("radius", "shape")]:
        some = gpu.download(pick)
        assert sorted(some) == sorted(pick)
        for k in pick:
            assert np.array_equal(some[k], every[k]), (pick, k)
    back = WorldBatch(scene.counts, form=form, plane=scene.plane)
    back.upload(**every)
    again = back.download(FIELDS)
    for k in FIELDS:
        assert np.array_equal(again[k], every[k]), k


@pytest.mark.parametrize("form", [0, 1])
def test_damping_by_body(form, cuda_lib):
    from cubez_gb300.batch import WorldBatch
    scene = scenes.precision(num_worlds=3, bodies=20, seed=9)
    rng = np.random.default_rng(9)
    scene.linear_damping[:] = rng.choice([0.95, 0.5, 1.0, 0.0, -0.0], scene.num_bodies)
    scene.angular_damping[:20] = 0.9
    scene.angular_damping[20:] = rng.uniform(0.1, 1.0, 40)
    gpu = WorldBatch.from_scene(scene, form=form)
    ref = OracleBatch(scene, form=ORC_FP64 if form == 0 else ORC_FP32)
    for dt in (DT, 0.01, DT):
        gpu.integrate(dt)
        ref.integrate(dt)
        g, r = gpu.download(("position", "velocity", "rotation")), ref.bodies()
        for k in g:
            assert np.array_equal(g[k], r[k]), k
