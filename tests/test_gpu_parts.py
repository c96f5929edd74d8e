"""Rollouts of 128 worlds or more run as parallel branches of their graph, each
over its own worlds (part_rule in cz_api.cu): the same bits as the phases
called one after the other over the whole batch, with empty worlds, worlds of
more than 64 bodies, odd counts, rollouts longer than one graph holds, and the
learned warm start."""
import numpy as np
import pytest

from cubez_gb300 import scenes

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0
FIELDS = ("position", "orientation", "velocity", "rotation", "motion", "is_awake", "inverse_inertia_world",
          "last_frame_acceleration")


def _scene(worlds, seed):
    parts = [scenes.mixed(num_worlds=worlds, seed=seed, min_bodies=1, max_bodies=24)]
    parts.append(scenes.piles(num_worlds=3, seed=seed, nx=5, nz=4, ny=4))
    counts = [int(c) for p in parts for c in p.counts]
    for at in (0, worlds // 2, len(counts)):
        counts.insert(at, 0)
    return scenes.Scene.concat(parts, counts=counts)


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("worlds,frames", [(122, 3), (127, 35), (700, 33)])
def test_parts_equal_the_phases(form, worlds, frames, cuda_lib):
    from cubez_gb300.batch import WorldBatch
    scene = _scene(worlds, 70 + worlds)
    scene.can_sleep[::3] = 1
    a = WorldBatch.from_scene(scene, form=form)
    b = WorldBatch.from_scene(scene, form=form)
    for _ in range(2):  # the second rollout starts from sorted queues
        a.step(frames, DT)
        for _ in range(frames):
            b.integrate(DT)
            b.narrowphase()
            b.resolve(DT)
    x, y = a.download(FIELDS), b.download(FIELDS)
    for k in FIELDS:
        assert np.array_equal(x[k], y[k]), k
    assert np.array_equal(a.contact_counts(), b.contact_counts())
    sa, sb = a.stats(), b.stats()
    for k in sa:
        assert np.array_equal(sa[k], sb[k]), k
    assert a.counters() == b.counters()


def test_parts_with_the_warm_start_equal_the_phases(cuda_lib):
    from cubez_gb300.batch import FORM_FP32, WorldBatch
    from cubez_gb300.learned import BLOB, OFF_B4, OFF_IS, OFF_OS, set_warm_start
    scene = scenes.precision(num_worlds=300, seed=79)
    blob = np.zeros(BLOB, np.float32)
    blob[OFF_IS:OFF_IS + 18] = 1.0
    blob[OFF_OS:OFF_OS + 3] = 1.0
    blob[OFF_B4] = 0.5
    batches = []
    for _ in range(2):
        b = WorldBatch.from_scene(scene, form=FORM_FP32)
        set_warm_start(b, blob)
        batches.append(b)
    a, b = batches
    a.step(120, DT)
    for _ in range(120):
        b.integrate(DT)
        b.narrowphase()
        b.resolve(DT)
    x, y = a.download(FIELDS), b.download(FIELDS)
    for k in FIELDS:
        assert np.array_equal(x[k], y[k]), k
    ca, cb = a.counters(), b.counters()
    assert ca["warm_worlds"] > 0
    for k in ("contacts", "vel_iterations", "warm_worlds", "warm_bodies", "warm_fallbacks"):
        assert ca[k] == cb[k], k
