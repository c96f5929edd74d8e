"""Which resolver a batch runs (wide_rule in cz_api.cu), as cz_batch_info
reports it."""
import numpy as np
import pytest

from cubez_gb300 import scenes

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0
FIELDS = ("position", "orientation", "velocity", "rotation", "motion", "is_awake")


@pytest.mark.parametrize("form", [0, 1])
def test_info_reports_the_launch(form, cuda_lib):
    from cubez_gb300.batch import WorldBatch
    few = WorldBatch([62] * 40, form=form)
    info = few.info()
    # four warps to a world, in a tile of eight contacts a body slot with their friction matrices
    assert info["resolver_ctas"] == 40
    assert info["resolver_smem"] >= 8 * 64 * (20 + 16) * info["real_bytes"]
    many = WorldBatch([62] * (7 * info["sms"] + 1), form=form)
    assert many.info()["resolver_smem"] != info["resolver_smem"]


@pytest.mark.parametrize("form", [0, 1])
def test_ctas_per_sm_bounds_the_launch(form, cuda_lib):
    """resolver_ctas_per_sm holds where four warps share a world, too; a CTA
    then takes several worlds, with the same bits."""
    from cubez_gb300.batch import WorldBatch
    sms = WorldBatch([1], form=form).info()["sms"]
    scene = scenes.mixed(num_worlds=2 * sms + 5, seed=8, min_bodies=40, max_bodies=62)
    a, b = (WorldBatch.from_scene(scene, form=form) for _ in range(2))
    b.set_tuning(resolver_ctas_per_sm=1)
    assert a.info()["resolver_smem"] == b.info()["resolver_smem"]
    assert a.info()["resolver_ctas"] == scene.num_worlds and b.info()["resolver_ctas"] == sms
    a.step(60, DT)  # in parts
    for _ in range(60):
        b.integrate(DT)
        b.narrowphase()
        b.resolve(DT)
    x, y = a.download(FIELDS), b.download(FIELDS)
    for k in FIELDS:
        assert np.array_equal(x[k], y[k]), k
    assert a.counters() == b.counters()


@pytest.mark.parametrize("form", [0, 1])
def test_reported_tuning_set_again_changes_nothing(form, cuda_lib):
    from cubez_gb300.batch import WorldBatch
    for worlds in (1, 40, 200, 311):
        b = WorldBatch([62] * worlds, form=form)
        before = b.info()
        b.set_tuning(**b.get_tuning())
        assert b.info() == before, worlds
