"""The leaf phase of the edits against the oracle where its lanes, lerps and source lookups can go wrong:
noise cells around the 4-voxel leaf and the 16-bit fraction, off-grid and partial footprints, copies whose
source box straddles leaves, leaves the grid below zero or overlaps its destination."""
import pytest

from gpu_util import gpu_canon

pytestmark = pytest.mark.gpu

LEVELS = 7
SCENE = dict(seed=3, octaves=4, num_materials=8, min_height_pct=30, max_height_pct=75, num_structures=0, structure_seed=0)


def check(svdag_lib, oracle_mod, edits):
    g = svdag_lib.MyGPUHashDAG(LEVELS, pool_bytes=1 << 28)
    g.build_terrain(**SCENE)
    o = oracle_mod.OracleDag(LEVELS)
    o.build_terrain(oracle_mod.TerrainParams(**SCENE))
    for e in edits:
        oe = oracle_mod.Edit()
        oe.tool, oe.material, oe.radius = e.tool, e.material, e.radius
        oe.center[:], oe.src[:], oe.dst[:] = list(e.center), list(e.src), list(e.dst)
        oe.noise_seed, oe.noise_cell_log2 = e.noise_seed, e.noise_cell_log2
        g.edit(e)
        st = o.edit(oe)
        got = g.last_edit_stats()
        assert got.edited_voxels == st.edited_voxels and list(got.svo_nodes) == list(st.svo_nodes)
        assert got.unique_items == st.unique_items
        assert gpu_canon(oracle_mod, g) == o.canon()
    g.free()


@pytest.mark.parametrize("cell_log2", [0, 1, 2, 3, 5, 15, 16, 17, 20])
def test_noise_paint_cells(svdag_lib, oracle_mod, cell_log2):
    import svdag.workloads as w

    check(svdag_lib, oracle_mod, [
        w.make_edit(svdag_lib.TOOL_BOX_PAINT_NOISE, 0, (60.0, 62.0, 57.0), 33.0, noise_seed=17, noise_cell_log2=cell_log2),
        w.make_edit(svdag_lib.TOOL_BOX_PAINT_NOISE, 0, (3.5, 50.25, 120.0), 20.75, noise_seed=5, noise_cell_log2=cell_log2)])


@pytest.mark.parametrize("offset", [(0, 0, 0), (1, 2, 3), (-7, 0, 5), (40, -3, 0), (-70, 4, -66)])
@pytest.mark.parametrize("radius", [1.0, 6.5, 19.0])
def test_copies(svdag_lib, oracle_mod, offset, radius):
    import svdag.workloads as w

    src = (50.0, 64.0, 48.0)
    dst = tuple(a + b for a, b in zip(src, offset))
    check(svdag_lib, oracle_mod, [
        w.make_edit(svdag_lib.TOOL_COPY, 0, src, radius, src=src, dst=dst),
        w.make_edit(svdag_lib.TOOL_COPY, 0, (4.0, 60.0, 3.0), radius, src=(4.0, 60.0, 3.0), dst=(30.0, 58.0, 35.0))])


@pytest.mark.parametrize("radius", [0.0, 0.7, 2.0, 9.3, 30.0])
@pytest.mark.parametrize("center", [(64.0, 60.0, 64.0), (61.5, 63.25, 1.75)])
def test_every_tool_on_and_off_the_grid(svdag_lib, oracle_mod, radius, center):
    import svdag.workloads as w

    s = svdag_lib
    check(svdag_lib, oracle_mod, [w.make_edit(t, 5, center, radius, noise_seed=13) for t in
                                  (s.TOOL_SPHERE_PAINT, s.TOOL_SPHERE_ERODE, s.TOOL_BOX_REMOVE, s.TOOL_SPHERE_ADD, s.TOOL_SPHERE_ERODE,
                                   s.TOOL_BOX_ADD, s.TOOL_SPHERE_REMOVE)])
