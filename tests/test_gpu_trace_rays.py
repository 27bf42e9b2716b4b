"""Primary rays where the traversal's shortcuts could differ from the oracle: directions with zero and
tiny components (their inverses are infinite or huge), cameras on node planes, inside, outside and far from
the grid, at depths 4 to 17, images of odd and single-pixel sizes."""
import ctypes

import numpy as np
import pytest

from gpu_util import gpu_trace

pytestmark = pytest.mark.gpu

VIEWS = {  # camera and target in units of the grid
    "axis": ((0.5, 0.9, 0.5), (0.5, 0.5, 0.5)),
    "axis_x": ((-0.25, 0.5, 0.5), (0.75, 0.5, 0.5)),
    "oblique": ((0.1, 0.95, 0.2), (0.7, 0.4, 0.6)),
    "nearly_axis": ((0.5, 0.8, 0.25), (0.5 + 1e-9, 0.8 - 1e-12, 0.75)),
    "outside": ((-3.0, 2.0, -2.5), (0.5, 0.5, 0.5)),
    "away": ((0.5, 0.9, 0.5), (0.4, 3.0, 0.6)),
}


@pytest.fixture(scope="module", params=[4, 9, 17])
def scene(request, svdag_lib, oracle_mod):
    import svdag.workloads as w

    levels = request.param
    g = svdag_lib.MyGPUHashDAG(levels, pool_bytes=4 << 30)
    o = oracle_mod.OracleDag(levels)
    if levels < 17:
        terrain = dict(seed=2, octaves=2, num_materials=8, min_height_pct=35, max_height_pct=70, num_structures=0, structure_seed=0)
        g.build_terrain(**terrain)
        o.build_terrain(oracle_mod.TerrainParams(**terrain))
    else:  # one sphere and one box in an empty grid of the full depth
        n = float(1 << levels)
        for tool, radius, x in ((svdag_lib.TOOL_SPHERE_ADD, 90.0, 0.5), (svdag_lib.TOOL_BOX_ADD, 64.0, 0.501)):
            e = w.make_edit(tool, 3, (x * n, 0.5 * n, 0.5 * n), radius)
            oe = oracle_mod.Edit()
            oe.tool, oe.material, oe.radius = e.tool, e.material, e.radius
            oe.center[:] = list(e.center)
            g.edit(e)
            o.edit(oe)
        g.sync()
    yield levels, g, o
    g.free()


@pytest.mark.parametrize("view", sorted(VIEWS))
@pytest.mark.parametrize("size", [(1, 1), (33, 9), (65, 31)])
def test_hits_equal_the_oracle(svdag_lib, oracle_mod, scene, view, size):
    levels, g, o = scene
    n = float(1 << levels)
    camera, target = ([v * n for v in p] for p in VIEWS[view])
    p = svdag_lib.get_trace_params(camera, target, *size)
    po = oracle_mod.TraceParams()
    for f in ("camera", "ray_min", "ray_ddx", "ray_ddy"):
        getattr(po, f)[:] = list(getattr(p, f))
    po.width, po.height = size
    got, want = gpu_trace(svdag_lib, g, p), o.trace(po)
    assert np.array_equal(got["path"], want["path"])
    hit = np.any(got["path"] != 0, axis=1)
    assert np.array_equal(got["material"][hit], want["material"][hit])
    for f in ("position", "normal", "dpdu", "dpdv"):  # the same IEEE operations: the same floats
        assert np.array_equal(got[f], want[f], equal_nan=True), f


@pytest.mark.parametrize("size", [(33, 4), (32, 4), (65, 8), (8, 65), (1, 1)])
def test_shading_of_both_pixel_orders(svdag_lib, oracle_mod, scene, size):
    """Images on both sides of the rule that gives a warp a row or a tile of pixels: sun visibility and
    ambient occlusion equal the oracle's for every pixel, none is left out."""
    import torch

    levels, g, o = scene
    n = float(1 << levels)
    p = svdag_lib.get_trace_params([0.1 * n, 0.95 * n, 0.2 * n], [0.7 * n, 0.4 * n, 0.6 * n], *size)
    po = oracle_mod.TraceParams()
    for f in ("camera", "ray_min", "ray_ddx", "ray_ddy"):
        getattr(po, f)[:] = list(getattr(p, f))
    po.width, po.height = size
    sh = svdag_lib.shade_params(levels, shadows=True, ao_samples=2, ao_ray_length=8.0)
    so = oracle_mod.ShadeParams()
    ctypes.memmove(ctypes.addressof(so), ctypes.addressof(sh), ctypes.sizeof(so))
    tracer = svdag_lib.DAGTracer(*size)
    tracer.resolve_paths(p, g)
    colors, sun, ao = tracer.resolve_lighting(p, g, sh, want_surfaces=True)
    torch.cuda.synchronize()
    want = o.shade(po, so, o.trace(po))
    assert np.array_equal(sun.cpu().numpy(), want[2])
    assert np.array_equal(ao.cpu().numpy(), want[3])
