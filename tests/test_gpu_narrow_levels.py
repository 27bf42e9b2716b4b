"""The launch forms of an edit where their dispatch can go wrong: footprints whose levels cross the
narrow limit (128 items) at every height, lie at the grid's corners, across or outside its faces, or
cover it. The chain of launches, one launch per phase and the persistent kernel must leave the same
DAG and counters, equal to the oracle's."""
import pytest

from gpu_util import gpu_canon

pytestmark = pytest.mark.gpu

LEVELS = 9
SCENE = dict(seed=1, octaves=4, num_materials=8, min_height_pct=35, max_height_pct=70, num_structures=8, structure_seed=2)
CENTERS = [(256.0, 250.0, 256.0), (0.0, 200.0, 511.0), (130.5, 240.25, -60.0)]


@pytest.mark.parametrize("radius", [0.0, 3.0, 11.0, 43.0, 90.0, 400.0])
@pytest.mark.parametrize("center", CENTERS)
def test_forms_agree(svdag_lib, oracle_mod, center, radius):
    import svdag.workloads as w

    s = svdag_lib
    tools = [s.TOOL_SPHERE_PAINT, s.TOOL_SPHERE_REMOVE, s.TOOL_COPY, s.TOOL_BOX_ADD, s.TOOL_BOX_PAINT_NOISE, s.TOOL_SPHERE_ADD]
    if radius <= 90.0:
        tools += [s.TOOL_SPHERE_ERODE, s.TOOL_MOVE, s.TOOL_BOX_REMOVE]
    forms = [s.MyGPUHashDAG(LEVELS, pool_bytes=1 << 30, scratch_bytes=1 << 29, **kw)
             for kw in ({}, {"phase_kernels": True}, {"persistent": True})]
    o = oracle_mod.OracleDag(LEVELS)
    o.build_terrain(oracle_mod.TerrainParams(**SCENE))
    for g in forms:
        g.build_terrain(**SCENE)
    dst = (center[0] + 37.0, center[1] - 9.0, center[2] + 1.0)
    for tool in tools:
        e = w.make_edit(tool, 6, center, radius, src=center, dst=dst, noise_seed=13, noise_cell_log2=3)
        oe = oracle_mod.Edit()
        oe.tool, oe.material, oe.radius = e.tool, e.material, e.radius
        oe.center[:], oe.src[:], oe.dst[:] = list(e.center), list(e.src), list(e.dst)
        oe.noise_seed, oe.noise_cell_log2 = e.noise_seed, e.noise_cell_log2
        st = o.edit(oe)
        for g in forms:
            g.edit(e)
            g.sync()
            if tool == s.TOOL_MOVE:
                continue  # two edits: the last counters are the paste's alone, the oracle's are both
            got = g.last_edit_stats()
            assert list(got.svo_nodes) == list(st.svo_nodes)
            assert (got.edited_voxels, got.unique_items, got.new_items) == (st.edited_voxels, st.unique_items, st.new_items)
        want = o.canon()
        for g in forms:
            assert gpu_canon(oracle_mod, g) == want
    for g in forms:
        g.undo()
        g.free()
