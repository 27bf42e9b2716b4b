"""Space that appending overflow slabs takes from the pool, by the growth of the regions' bump pointers
over the call. With 1 and 32 lanes a key one slab is taken per append, so a table grows by exactly the
slabs of its chains. With 2 to 16 lanes a group that loses the race for a link keeps its slab for its
next append, so keys of one size class leave at most one unused slab a group of the launch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SLAB_BYTES = 32 + 24 * 4 * 4  # a header and 24 slots of three words, padded to four


@pytest.mark.parametrize("op", ["add", "find_or_add"])
@pytest.mark.parametrize("lanes", [1, 4, 8, 16, 32])
def test_pool_bytes_of_full_buckets(svdag_lib, op, lanes):
    import torch

    n, buckets = 1 << 20, 64
    dag = svdag_lib.MyGPUHashDAG(6, pool_bytes=3 << 30)
    table = dag.create_table(svdag_lib.KIND_NODE, [0, buckets] + [0] * 7)
    words = torch.empty((n, 3), dtype=torch.int32, device="cuda")
    words[:, 0] = 0b101  # two children: keys of three words
    words[:, 1] = torch.arange(n, device="cuda")
    words[:, 2] = 7
    offs = torch.arange(0, 3 * n, 3, dtype=torch.int32, device="cuda")
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    before = dag.stats().item_region_used_bytes
    getattr(table, op)(words.reshape(-1), offs, n, 3 * n, out, lanes=lanes)
    dag.sync()
    st = table.stats()
    assert st.items == n
    slabs = (dag.stats().item_region_used_bytes - before) / SLAB_BYTES
    groups = min(n, torch.cuda.get_device_properties(0).multi_processor_count * 8 * 256 // lanes)
    if lanes in (1, 32):
        assert slabs == st.overflow_slabs
    else:
        assert st.overflow_slabs <= slabs <= st.overflow_slabs + groups
    got = torch.empty((n, 10), dtype=torch.int32, device="cuda")
    table.read(out, n, got)
    assert torch.equal(got[:, :3], words)
    dag.free()
