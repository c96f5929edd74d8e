"""The narrowphase's tests spread over lanes (np_flush in cz_kernels.cuh): a
cube's half-space vertices on eight lanes each, a cube pair's axes on sixteen,
one set of axes for both orders of a pair.  Contact lists against the oracle,
bit for bit, where a chunk holds more cubes or pairs than one pass of the CTA
takes, for every CTA size, and for callers' lists with repeated and reversed
tests."""
import numpy as np
import pytest

from cubez_gb300 import scenes
from oracle.oracle import FP32 as ORC_FP32
from oracle.oracle import FP64 as ORC_FP64
from oracle.oracle import OracleBatch

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


def _packed(seed, offsets=False):
    """Worlds of 1 to 64 cubes and spheres, packed close and low: most cubes
    reach the half-space and several others."""
    scene = scenes.mixed(num_worlds=12, seed=seed, min_bodies=1, max_bodies=64)
    rng = np.random.default_rng(seed)
    scene.position[:, (0, 2)] *= 0.35
    scene.position[:, 1] = rng.uniform(0.0, 1.5, scene.num_bodies)
    flip = rng.random(scene.num_bodies) < 0.6  # more cubes than spheres
    scene.shape = np.where(flip, scenes.CUBE, scene.shape).astype(np.int32)
    scene.half_size = np.where((scene.shape == scenes.CUBE)[:, None] & (scene.half_size == 0), 0.5, scene.half_size)
    # some exactly axis-aligned cubes: equal penetrations on several axes
    still = rng.random(scene.num_bodies) < 0.3
    scene.orientation[still] = (1.0, 0.0, 0.0, 0.0)
    scene.half_size[still & (scene.shape == scenes.CUBE)] = 0.5
    if offsets:
        scene.collider_offset = scenes.offsets(num_worlds=1, bodies=scene.num_bodies, seed=seed).collider_offset
    return scene


def _check(gpu, ref, scene):
    total = 0
    counts = gpu.contact_counts()
    for w in range(scene.num_worlds):
        g, r = gpu.contacts(w), ref.contacts(w)
        assert counts[w] == len(r["penetration"]), w
        for k in ("bodies", "point", "normal", "penetration"):
            assert np.array_equal(g[k], r[k]), (w, k)
        total += counts[w]
    return total


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("threads", [32, 64, 128, 256])
@pytest.mark.parametrize("offsets", [False, True])
def test_packed_worlds_bit_exact(form, threads, offsets, cuda_lib):
    from cubez_gb300.batch import WorldBatch
    scene = _packed(90 + threads, offsets)
    gpu = WorldBatch.from_scene(scene, form=form)
    gpu.set_tuning(narrowphase_threads=threads)
    ref = OracleBatch(scene, form=ORC_FP64 if form == 0 else ORC_FP32)
    gpu.integrate(DT)
    ref.integrate(DT)
    gpu.narrowphase()
    ref.narrowphase()
    assert _check(gpu, ref, scene) > 1000


@pytest.mark.parametrize("form", [0, 1])
def test_callers_lists_bit_exact(form, cuda_lib):
    from cubez_gb300.batch import WorldBatch
    scene = _packed(99)
    w = int(np.argmax(scene.counts))
    n = int(scene.counts[w])
    gpu = WorldBatch.from_scene(scene, form=form)
    ref = OracleBatch(scene, form=ORC_FP64 if form == 0 else ORC_FP32)
    gpu.integrate(DT)
    ref.integrate(DT)
    rng = np.random.default_rng(5)
    for m in (1, 2, 255, 256, 257, 3000):
        i = rng.integers(0, n, m)
        j = rng.integers(-1, n - 1, m)
        j = np.where(j >= i, j + 1, j)  # -1 or another body
        units = np.stack([i, j], axis=1)
        units[m // 2:] = np.where(units[:m - m // 2, 1:] >= 0, units[:m - m // 2, ::-1], units[:m - m // 2])
        gpu.collide(w, units)
        ref.collide(w, units)
        g, r = gpu.contacts(w), ref.contacts(w)
        for k in ("bodies", "point", "normal", "penetration"):
            assert np.array_equal(g[k], r[k]), (m, k)
