"""Batches of up to three worlds per SM are resolved with four warps to a world
(k_resolve_wide): the same bits as the same worlds give in a larger batch, one
warp to a world, with budgets that run out, sleeping bodies, worlds of one to
many islands, empty worlds, and contact lists past the shared tile."""
import numpy as np
import pytest

from cubez_gb300 import scenes

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0
FIELDS = ("position", "orientation", "velocity", "rotation", "motion", "is_awake", "inverse_inertia_world",
          "last_frame_acceleration")


def _crowd(seed):
    """Worlds whose bodies all overlap: one island, more than 8 contacts a body."""
    s = scenes.mixed(num_worlds=4, seed=seed, min_bodies=24, max_bodies=30)
    s.position[:] = 0.02 * s.position + np.array([0.0, 0.6, 0.0])
    return s


def _scene(worlds, seed):
    parts = [scenes.mixed(num_worlds=worlds - 7, seed=seed, min_bodies=1, max_bodies=64), _crowd(seed)]
    counts = [int(c) for p in parts for c in p.counts]
    for at in (0, worlds // 2, len(counts)):
        counts.insert(at, 0)
    scene = scenes.Scene.concat(parts, counts=counts)
    scene.can_sleep[::3] = 1
    return scene


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("worlds,budget", [(8, 0), (40, 0), (150, 0), (400, 0), (700, 0), (40, 1), (40, 30), (40, 200)])
def test_wide_equals_one_warp_per_world(form, worlds, budget, cuda_lib):
    from cubez_gb300.batch import WorldBatch
    scene = _scene(worlds, 90 + worlds)
    filler = scenes.precision(num_worlds=1200, bodies=2, seed=5)
    both = scenes.Scene.concat([scene, filler])
    kw = {"form": form, "max_iterations": budget, "contact_capacity": 1024}
    a, b = WorldBatch.from_scene(scene, **kw), WorldBatch.from_scene(both, **kw)
    n = scene.num_bodies
    longest = 0
    for frames in (1, 49, 50, 50):  # (the crowds are apart after a few frames)
        a.step(frames, DT)
        longest = max(longest, int(a.contact_counts().max()))
        for _ in range(frames):  # the phases: one launch over all worlds
            b.integrate(DT)
            b.narrowphase()
            b.resolve(DT)
        x, y = a.download(FIELDS), b.download(FIELDS)
        for k in FIELDS:
            assert np.array_equal(x[k], y[k][:n]), k
        sa, sb = a.stats(), b.stats()
        for k in sa:
            assert np.array_equal(sa[k], sb[k][:worlds]), k
    assert longest > 8 * 30


@pytest.mark.parametrize("form", [0, 1])
def test_wide_writes_the_contacts_back(form, cuda_lib):
    from cubez_gb300.batch import WorldBatch
    scene = _scene(12, 33)
    both = scenes.Scene.concat([scene, scenes.precision(num_worlds=600, bodies=2, seed=5)])
    a, b = WorldBatch.from_scene(scene, form=form), WorldBatch.from_scene(both, form=form)
    for _ in range(40):
        for g in (a, b):
            g.integrate(DT)
            g.narrowphase()
            g.resolve(DT)
    for w in range(12):
        x, y = a.contacts(w), b.contacts(w)
        for k in x:
            assert np.array_equal(x[k], y[k]), (w, k)
