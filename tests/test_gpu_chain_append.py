"""Overflow slabs under contention: however many threads find a bucket full at once, each slab of
its chain is appended once, so a table of one bucket holds its n keys in exactly ceil(n / 24) slabs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SLOTS = 24


@pytest.mark.parametrize("lanes", [1, 2, 8, 32])
@pytest.mark.parametrize("n", [1, 24, 25, 49, 3001])
def test_one_bucket_chain_has_no_spare_slabs(svdag_lib, lanes, n):
    import torch

    dag = svdag_lib.MyGPUHashDAG(6, pool_bytes=1 << 26)
    table = dag.create_table(svdag_lib.KIND_NODE, [0, 1] + [0] * 7)
    rng = np.random.default_rng(n)
    words = rng.integers(0, 1 << 28, (n, 3)).astype(np.uint32)
    words[:, 0] = 0b101  # two children: keys of three words
    words[:, 1] = rng.permutation(n)
    flat = torch.from_numpy(words.reshape(-1).view(np.int32)).cuda()
    offs = torch.arange(0, 3 * n, 3, dtype=torch.int32, device="cuda")
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    table.add(flat, offs, n, 3 * n, out, lanes=lanes)
    dag.sync()
    st = table.stats()
    assert st.items == n
    assert st.overflow_slabs == (n + SLOTS - 1) // SLOTS - 1
    assert len(np.unique(out.cpu().numpy())) == n
    table.find(flat, offs, n, 3 * n, out, lanes=lanes)
    got = torch.empty((n, 10), dtype=torch.int32, device="cuda")
    table.read(out, n, got)
    dag.sync()
    assert np.array_equal(got.cpu().numpy().view(np.uint32)[:, :3], words)
    dag.free()


def test_a_level_table_starts_with_room_for_versions(svdag_lib):
    """The root of a scene is one item, but each edit adds a version of it: 60 edits fit the first
    slabs of the root's table, with no chain."""
    import svdag.workloads as w

    dag = svdag_lib.MyGPUHashDAG(10, pool_bytes=2 << 30)
    dag.build_terrain(**w.C0_TERRAIN)
    for tool, material, center, radius in w.c0_edits(60):
        dag.edit(w.make_edit(tool, material, center, min(radius, 12.0)))
    dag.sync()
    st = dag.table(0).stats()
    assert st.items > 30
    assert st.overflow_slabs == 0
    dag.free()
