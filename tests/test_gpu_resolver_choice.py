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
