"""The resolver with one warp per world (k_resolve with 32 lanes), which takes
batches of more than seven worlds per SM and worlds of up to a dozen bodies
(wide_rule in cz_api.cu): shared tiles of every size, records past the tile,
budgets that run out, and the caller's contacts written back, against the
oracle bit for bit.  Worlds of two bodies fill the batches up."""
import numpy as np
import pytest

from cubez_gb300 import scenes
from oracle.oracle import FP32 as ORC_FP32
from oracle.oracle import FP64 as ORC_FP64
from oracle.oracle import OracleBatch
from tests import test_gpu_api as api

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0
STATE = ("position", "orientation", "velocity", "rotation", "motion", "is_awake")


def _among_many(scene, sms):
    """The scene with as many small worlds behind it as one warp per world needs."""
    return scenes.Scene.concat([scene, scenes.precision(num_worlds=7 * sms + 1, bodies=2, seed=5)])


def _sms():
    from cubez_gb300.batch import WorldBatch
    return WorldBatch([1]).info()["sms"]


def _assert_state(gpu, ref, n):
    g, r = gpu.download(STATE), ref.bodies()
    for k in STATE:
        assert np.array_equal(g[k][:n], r[k]), k


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("bodies,tile", [(32, 96), (33, 128), (50, 160), (64, 192)])
def test_tiles_bit_exact(form, bodies, tile, cuda_lib):
    from cubez_gb300.batch import WorldBatch
    scene = scenes.precision(num_worlds=40, bodies=bodies, seed=31)
    both = _among_many(scene, _sms())
    ref = OracleBatch(scene, form=ORC_FP64 if form == 0 else ORC_FP32)
    ref.step(130, DT, threads=8)
    assert ref.stats()["contacts"].max() > 32
    bytes_of = []
    for choice in (0, 32):
        gpu = WorldBatch.from_scene(both, form=form)
        if choice:
            gpu.set_tuning(resolver_contacts=choice)
        assert gpu.get_tuning()["resolver_contacts"] == (choice or tile)
        bytes_of.append(gpu.info()["resolver_smem"])
        gpu.step(130, DT)
        _assert_state(gpu, ref, scene.num_bodies)
    assert bytes_of[0] != bytes_of[1]  # four warps to a world would take the same tile for both


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("budget", [1, 7, 33, 150, 4000])
def test_budgets_and_spilled_records_bit_exact(form, budget, cuda_lib):
    from cubez_gb300.batch import WorldBatch
    orc = ORC_FP64 if form == 0 else ORC_FP32
    scene = scenes.mixed(num_worlds=24, seed=51, min_bodies=1, max_bodies=64)
    scene.can_sleep[::3] = 1
    ref = OracleBatch(scene, form=orc)
    ref.step(130, DT, threads=8)
    st = ref.bodies()
    for k in STATE:
        setattr(scene, k, st[k])
    both = _among_many(scene, _sms())
    for tile in (32, 192):
        gpu = WorldBatch.from_scene(both, form=form, max_iterations=budget)
        gpu.set_tuning(resolver_contacts=tile)
        ref = OracleBatch(scene, form=orc)
        hit = 0
        for _ in range(3):
            gpu.integrate(DT)
            gpu.narrowphase()
            gpu.resolve(DT)
            ref.integrate(DT)
            ref.narrowphase()
            ref.resolve_fixed(budget, DT)
            _assert_state(gpu, ref, scene.num_bodies)
            gs, rs = gpu.stats(), ref.stats()
            for k in ("pos_iterations", "vel_iterations"):
                assert np.array_equal(gs[k][:scene.num_worlds], rs[k]), k
            hit += int((rs["vel_iterations"] >= budget).sum())
        assert rs["contacts"].max() > 32 and (hit > 0) == (budget < 4000)


# 12 bodies: one warp; 24: four warps.  The list once, and repeated until it
# exceeds either kernel's shared tile.
@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("seed,bodies,contacts", [(31, 12, 0), (31, 12, 150), (55, 24, 0), (55, 24, 500)])
def test_contacts_written_back(form, seed, bodies, contacts, cuda_lib):
    scene, c = api.scene_with_contacts(seed, bodies, 150, form)
    n = len(c["penetration"])
    assert n > 8
    rng = np.random.default_rng(bodies)
    at = np.arange(max(contacts, n)) % n
    c = {k: c[k][at] for k in c}
    if contacts:
        c["point"] = c["point"] + rng.normal(0.0, 0.01, c["point"].shape)
        c["penetration"] = c["penetration"] + rng.uniform(0.0, 0.01, len(at))
    # half-space contacts given with body 0 nil, as calculateInternals swaps them (contact.go:61-65)
    nil = (c["bodies"][:, 1] < 0) & (rng.random(len(at)) < 0.5)
    assert nil.any()
    c["bodies"][nil] = c["bodies"][nil][:, ::-1]
    c["normal"][nil] *= -1.0
    for budget in (4 * len(at), 40):
        st, arrays, arr, ref = api.resolve_both(scene, c, budget, form)
        assert st == 0, cuda_lib.cz_last_error()
        assert ref.stats()["pos_iterations"][0] > 0 and ref.stats()["vel_iterations"][0] > 0
        assert all(a.body[0] >= 0 for a in arr)
        api.assert_matches_oracle(arrays, arr, ref)
