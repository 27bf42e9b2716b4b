"""Find-or-add with every lane count over keys of all sizes in few buckets, so that inserts fill slabs,
append others and walk past them: one copy per distinct key, the same handles from a second call that
finds all of them, and from a search."""
import numpy as np
import pytest

from test_gpu_tables import dev, key_list, leaf_keys, node_keys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes", [1, 2, 4, 8, 16, 32])
@pytest.mark.parametrize("kind", [0, 1])
def test_find_or_add_grows_chains(svdag_lib, lanes, kind):
    import torch

    rng = np.random.default_rng(500 + lanes + 7 * kind)
    n = 12000
    dag = svdag_lib.MyGPUHashDAG(6, pool_bytes=1 << 28)
    words, offs = (node_keys if kind == 0 else leaf_keys)(rng, n)
    distinct = len(set(key_list(words, offs)))
    table = dag.create_table(kind, [11] * 9)
    first = torch.empty(n, dtype=torch.int32, device="cuda")
    half = n // 2  # the first half alone, then all keys: found and new ones side by side in a warp
    table.find_or_add(dev(words[: offs[half]]), dev(offs[:half]), half, int(offs[half]), first, lanes=lanes)
    table.find_or_add(dev(words), dev(offs), n, len(words), first, lanes=lanes)
    again, found = torch.empty_like(first), torch.empty_like(first)
    table.find_or_add(dev(words), dev(offs), n, len(words), again, lanes=lanes)
    table.find(dev(words), dev(offs), n, len(words), found, lanes=lanes)
    out = torch.empty((n, 10), dtype=torch.int32, device="cuda")
    table.read(first, n, out)
    dag.sync()
    st = table.stats()
    assert st.items == distinct
    assert st.overflow_slabs > 0
    assert torch.equal(first, again) and torch.equal(first, found)
    got = out.cpu().numpy().view(np.uint32)
    assert all(tuple(got[i][: len(k)]) == tuple(k) for i, k in enumerate(key_list(words, offs)))
    dag.free()
