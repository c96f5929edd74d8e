"""The resolver's contact tile follows the worlds' body slots (tile_rule in
cz_api.cu): the same bits as with the smallest tile, and a caller's own choice
stays."""
import numpy as np
import pytest

from cubez_gb300 import scenes

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0
FIELDS = ("position", "orientation", "velocity", "rotation", "motion", "is_awake")


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("bodies,tile", [(4, None), (32, 96), (33, 128), (50, 160), (64, 192)])
def test_tile_by_bodies(form, bodies, tile, cuda_lib):
    from cubez_gb300.batch import WorldBatch
    scene = scenes.precision(num_worlds=200, bodies=bodies, seed=31)
    a, b, c = (WorldBatch.from_scene(scene, form=form) for _ in range(3))
    if tile:
        assert a.get_tuning()["resolver_contacts"] == tile
    b.set_tuning(resolver_contacts=32)
    c.set_tuning(resolver_lanes=16)
    assert b.get_tuning()["resolver_contacts"] == 32 and c.get_tuning()["resolver_contacts"] <= 96
    for g in (a, b, c):
        g.step(130, DT)
    x = a.download(FIELDS)
    for g in (b, c):
        y = g.download(FIELDS)
        for k in FIELDS:
            assert np.array_equal(x[k], y[k]), k
