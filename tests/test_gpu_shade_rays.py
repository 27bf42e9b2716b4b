"""Shadow and ambient-occlusion rays whose origin is not an ordinary point: a hit buffer may hold positions
with NaN or infinite components (a record of a ray whose own arithmetic overflowed, or a caller's own
records). Sun visibility and occlusion equal the oracle's for every combination of axes."""
import ctypes
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LEVELS = 8


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 1e38, -3e38])
def test_origins_off_the_number_line(svdag_lib, oracle_mod, value):
    import torch

    terrain = dict(seed=2, octaves=3, num_materials=8, min_height_pct=35, max_height_pct=70, num_structures=6, structure_seed=1)
    g = svdag_lib.MyGPUHashDAG(LEVELS, pool_bytes=1 << 28)
    o = oracle_mod.OracleDag(LEVELS)
    g.build_terrain(**terrain)
    o.build_terrain(oracle_mod.TerrainParams(**terrain))
    p = svdag_lib.get_trace_params((25.0, 240.0, 50.0), (180.0, 100.0, 150.0), 96, 64)
    po = oracle_mod.TraceParams()
    for f in ("camera", "ray_min", "ray_ddx", "ray_ddy"):
        getattr(po, f)[:] = list(getattr(p, f))
    po.width, po.height = p.width, p.height
    tracer = svdag_lib.DAGTracer(p.width, p.height)
    tracer.resolve_paths(p, g)
    hits = tracer.hits_numpy().copy()
    axes = [c for n in (0, 1, 2, 3) for c in itertools.combinations(range(3), n)]
    for i in range(len(hits)):
        for a in axes[(i + i // p.width) % len(axes)]:
            hits["position"][i, a] = value
    tracer.hits.copy_(torch.from_numpy(hits.view(np.uint8).reshape(-1)))
    shade = svdag_lib.shade_params(LEVELS, shadows=True, ao_samples=3, ao_ray_length=20.0)
    so = oracle_mod.ShadeParams()
    ctypes.memmove(ctypes.addressof(so), ctypes.addressof(shade), ctypes.sizeof(so))
    _, sun, ao = tracer.resolve_lighting(p, g, shade, want_surfaces=True)
    g.sync()
    _, _, want_sun, want_ao = o.shade(po, so, hits)
    assert np.any(hits["path"] != 0, axis=1).mean() > 0.3
    assert np.array_equal(sun.cpu().numpy(), want_sun, equal_nan=True)
    assert np.array_equal(ao.cpu().numpy(), want_ao, equal_nan=True)
    g.free()
