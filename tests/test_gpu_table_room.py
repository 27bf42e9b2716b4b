"""Level tables start with room for versions of the upper nodes, but only with space that their scene does
not need: a scene that fits its pool with tables of the counted sizes still builds and loads there."""
import math

import numpy as np
import pytest

from gpu_util import gpu_canon

pytestmark = pytest.mark.gpu

# Three items in four lie in overflow slabs, whose number a whole scene's buckets fix to a fraction of a percent;
# the scratch arena is one in which the scene is built in one piece.
LEVELS, LOAD, SCRATCH = 12, 48, 5 << 30
SCENE = dict(seed=4, octaves=6, num_materials=8, min_height_pct=35, max_height_pct=70, num_structures=16, structure_seed=7)
BODY_WORDS = [24 * ((k + 3) // 4 * 4) for k in range(2, 11)]


def expected_overflow(items, buckets):
    """Overflow slabs of `items` items hashed to `buckets` buckets, 24 a slab (a Poisson count a bucket)."""
    if not items:
        return 0.0
    mean = items / buckets
    x = np.arange(int(mean + 12 * math.sqrt(mean) + 30))
    p = np.exp(-mean + x * math.log(mean) - np.array([math.lgamma(v + 1) for v in x]))
    return buckets * float((p * np.maximum(0, np.ceil(x / 24) - 1)).sum())


def new_dag(svdag_lib, pool):
    return svdag_lib.MyGPUHashDAG(LEVELS, pool_bytes=pool, scratch_bytes=SCRATCH, load_factor=LOAD)


@pytest.fixture(scope="module")
def scene(svdag_lib, oracle_mod):
    """(canonical DAG, snapshot, pool bytes for the scene's tables, the expected overflow slabs and 0.6 % more of
    those)."""
    g = new_dag(svdag_lib, SCRATCH + (384 << 20))
    g.build_terrain(**SCENE)
    words = overflow = 0
    for level in range(LEVELS - 1):
        _, items = g.export_level(level)
        if level == LEVELS - 2:
            voxels = np.bitwise_count(items[:, 0]).astype(int) + np.bitwise_count(items[:, 1]).astype(int)
            size = 2 + (4 * voxels + 31) // 32
        else:
            size = 1 + np.bitwise_count(items[:, 0] & 0xFF).astype(int)
        for n, w in zip(np.bincount(size - 2, minlength=9), BODY_WORDS):
            want = -(-(int(n) + 16) // LOAD)  # sixteen more: the canonical items are counted in every class
            words += want * w
            overflow += expected_overflow(int(n), want) * w
    assert overflow > words
    # the item region is twelve thirteenths of what the other regions leave: solve for the pool by its reported size
    pool = SCRATCH + (256 << 20)
    tight = new_dag(svdag_lib, pool)
    pool += int(4 * (words + 1.006 * overflow) * 13 / 12) + 8192 - tight.stats().item_region_bytes
    tight.free()
    out = gpu_canon(oracle_mod, g), g.save_items(), pool
    g.free()
    return out


def test_a_scene_that_just_fits_builds(svdag_lib, oracle_mod, scene):
    canon, _, pool = scene
    g = new_dag(svdag_lib, pool)
    g.build_terrain(**SCENE)
    g.sync()
    assert gpu_canon(oracle_mod, g) == canon
    g.free()


def test_a_snapshot_that_just_fits_loads(svdag_lib, oracle_mod, scene):
    canon, snap, pool = scene
    g = new_dag(svdag_lib, pool)
    g.load_items(snap)
    assert gpu_canon(oracle_mod, g) == canon
    g.free()


def test_a_roomy_pool_has_the_minimum(svdag_lib):
    g = svdag_lib.MyGPUHashDAG(8, pool_bytes=8 << 30)
    g.build_terrain(seed=4, octaves=3, num_materials=8, min_height_pct=35, max_height_pct=70)
    assert g.table(0).stats().buckets == 9 * 2048
    g.free()
