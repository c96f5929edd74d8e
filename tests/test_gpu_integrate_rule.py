"""Integrate's launch shape (integrate_cta in cz_api.cu, integrate_as in
cz_form_impl.cuh) follows the batch's bodies, in one launch or in parts, and a
caller's own CTA size holds at every batch size; the bits are the same."""
import numpy as np
import pytest

from cubez_gb300 import scenes

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0
FIELDS = ("position", "orientation", "velocity", "rotation", "motion", "is_awake", "inverse_inertia_world")


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("worlds,bodies,cta", [(1, 1, 32), (7, 9, 32), (130, 30, 32), (520, 32, 32), (1024, 32, 32),
                                               (1030, 32, 256), (40, 300, 32)])
def test_cta_size(form, worlds, bodies, cta, cuda_lib):
    from cubez_gb300.batch import WorldBatch
    scene = scenes.precision(num_worlds=worlds, bodies=bodies, seed=worlds)
    scene.can_sleep[::3] = 1
    by_rule = WorldBatch.from_scene(scene, form=form)
    assert by_rule.get_tuning()["integrate_threads"] == cta
    by_rule.step(4, DT)
    want = by_rule.download(FIELDS)
    for threads in (32, 96, 256):
        b = WorldBatch.from_scene(scene, form=form)
        b.set_tuning(integrate_threads=threads)
        assert b.get_tuning()["integrate_threads"] == threads
        for _ in range(3):
            b.step(1, DT)
        b.integrate(DT)
        b.narrowphase()
        b.resolve(DT)
        got = b.download(FIELDS)
        for k in FIELDS:
            assert np.array_equal(got[k], want[k]), (threads, k)
