"""Edits that run alone in the one-block kernel (up to 400 estimated leaves in a context created for it), at
the sizes where its leaves are more than a narrow level holds (128) and at the smallest: every tool, across
node planes, at a corner and across a face of the grid. DAG and counters equal the oracle's, and the
kernel's phase stamps show that it ran."""
import pytest

from gpu_util import gpu_canon

pytestmark = pytest.mark.gpu

LEVELS = 9
SCENE = dict(seed=1, octaves=4, num_materials=8, min_height_pct=35, max_height_pct=70, num_structures=8, structure_seed=2)
CENTERS = [(256.0, 250.0, 256.0), (129.5, 241.25, 383.0), (2.0, 200.0, 509.0), (300.0, 255.0, -5.0)]


@pytest.mark.parametrize("radius", [0.0, 5.0, 10.0, 10.6])  # 10.6: 389 leaves estimated
@pytest.mark.parametrize("center", CENTERS)
def test_one_block_edits_match_the_oracle(svdag_lib, oracle_mod, center, radius):
    import svdag.workloads as w

    s = svdag_lib
    g = s.MyGPUHashDAG(LEVELS, pool_bytes=1 << 29, scratch_bytes=1 << 28, persistent=True)
    g.build_terrain(**SCENE)
    o = oracle_mod.OracleDag(LEVELS)
    o.build_terrain(oracle_mod.TerrainParams(**SCENE))
    dst = (center[0] + 21.0, center[1] - 9.0, center[2] + 1.0)
    last, most = [], 0
    for tool in (s.TOOL_SPHERE_PAINT, s.TOOL_BOX_PAINT_NOISE, s.TOOL_SPHERE_ERODE, s.TOOL_COPY, s.TOOL_BOX_REMOVE, s.TOOL_SPHERE_ADD,
                 s.TOOL_BOX_ADD, s.TOOL_SPHERE_REMOVE, s.TOOL_MOVE):
        e = w.make_edit(tool, 6, center, radius, src=center, dst=dst, noise_seed=13, noise_cell_log2=1)
        oe = oracle_mod.Edit()
        oe.tool, oe.material, oe.radius = e.tool, e.material, e.radius
        oe.center[:], oe.src[:], oe.dst[:] = list(e.center), list(e.src), list(e.dst)
        oe.noise_seed, oe.noise_cell_log2 = e.noise_seed, e.noise_cell_log2
        want = o.edit(oe)
        g.edit(e)
        g.sync()
        stamps = list(g.last_edit_phase_times())
        assert len(stamps) > 3 and stamps[0] > (last[-1] if last else 0)
        last = stamps
        assert gpu_canon(oracle_mod, g) == o.canon()
        if tool == s.TOOL_MOVE:
            continue  # two edits: the last counters are the paste's alone, the oracle's are both
        got = g.last_edit_stats()
        assert list(got.svo_nodes) == list(want.svo_nodes)
        assert (got.edited_voxels, got.unique_items, got.new_items) == (want.edited_voxels, want.unique_items, want.new_items)
        most = max(most, got.svo_nodes[LEVELS - 2])
    if radius > 10 and center == CENTERS[0]:
        assert most > 128  # a wide leaf level
    g.free()
