"""Parts of more than 256 worlds sort their own worlds by cost after every
frame (k_reorder over a part's slice of the queues, kReorderWorlds in
cz_api.cu): the same bits as the phases over the whole batch, plain and with
the learned warm start, with empty worlds and worlds of more than 64 bodies."""
import numpy as np
import pytest

from cubez_gb300 import _lib, scenes

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0
FIELDS = ("position", "orientation", "velocity", "rotation", "motion", "is_awake")


def _scene(worlds, bodies):
    parts = [scenes.precision(num_worlds=worlds // 2, bodies=bodies, seed=worlds),
             scenes.piles(num_worlds=2, seed=7, nx=5, nz=4, ny=4),
             scenes.precision(num_worlds=worlds - worlds // 2, bodies=bodies, seed=worlds + 1)]
    counts = [int(c) for p in parts for c in p.counts]
    for at in (0, worlds // 3, len(counts)):
        counts.insert(at, 0)
    scene = scenes.Scene.concat(parts, counts=counts)
    scene.position[::7, 1] += 0.5  # unlike work in the worlds
    return scene


@pytest.mark.parametrize("form,worlds,bodies,warm", [(1, 2100, 4, False), (1, 2100, 4, True), (0, 8300, 2, False)])
def test_sorted_parts_equal_the_phases(form, worlds, bodies, warm, cuda_lib):
    from cubez_gb300.batch import WorldBatch
    scene = _scene(worlds, bodies)
    batches = [WorldBatch.from_scene(scene, form=form) for _ in range(2)]
    if warm:
        from cubez_gb300.learned import BLOB, OFF_B4, OFF_IS, OFF_OS, set_warm_start
        blob = np.zeros(BLOB, np.float32)
        blob[OFF_IS:OFF_IS + 18] = 1.0
        blob[OFF_OS:OFF_OS + 3] = 1.0
        blob[OFF_B4] = 0.5
        for b in batches:
            set_warm_start(b, blob)
    a, b = batches
    parts = min(scene.num_worlds // 64, 8 if form else 32)
    for frames in (60, 3):  # on the ground, then from sorted queues
        a.prepare_rollout(frames, DT)
        before = _lib.kernel_launches()
        a.step(frames, DT)
        # integrate, narrowphase, resolve and the sort in every part, the piles' resolver in one or two,
        # the features with the warm start
        per_frame = (_lib.kernel_launches() - before) / frames
        assert per_frame in [parts * (5 if warm else 4) + big for big in (1, 2)]
        for _ in range(frames):
            b.integrate(DT)
            b.narrowphase()
            b.resolve(DT)
        x, y = a.download(FIELDS), b.download(FIELDS)
        for k in FIELDS:
            assert np.array_equal(x[k], y[k]), k
        sa, sb = a.stats(), b.stats()
        for k in sa:
            assert np.array_equal(sa[k], sb[k]), k
    ca, cb = a.counters(), b.counters()
    assert ca["contacts"] > 0 and ca["vel_iterations"] > 0
    assert (ca["warm_worlds"] > 0) == warm
    for k in ca:
        if k != "warm_scale_sum":  # (a sum of floats in any order)
            assert ca[k] == cb[k], k
