"""Reading table items back, whole blocks and remainders, at misaligned outputs: every word of a stored
key and zeros behind it, a row of zeros for a handle that names nothing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 1024 * 300 + 7])
@pytest.mark.parametrize("kind", [0, 1])
def test_read_rows(svdag_lib, kind, n):
    import torch

    rng = np.random.default_rng(n + kind)
    if kind == 0:  # nodes of 2..9 words
        counts = rng.integers(1, 9, n)
        head = ((1 << counts) - 1).astype(np.uint32)
        sizes = 1 + counts
    else:  # leaves of 3..10 words
        voxels = rng.integers(1, 65, n)
        sizes = 2 + (voxels * 4 + 31) // 32
    words = rng.integers(0, 1 << 32, (n, 10), dtype=np.uint64).astype(np.uint32)
    if kind == 0:
        words[:, 0] = head
    else:
        full = (1 << 32) - 1
        words[:, 0] = [full if v >= 32 else (1 << int(v)) - 1 for v in voxels]
        words[:, 1] = [full if v >= 64 else (1 << int(v - 32)) - 1 if v > 32 else 0 for v in voxels]
    words[np.arange(10)[None, :] >= sizes[:, None]] = 0
    flat = words[np.arange(10)[None, :] < sizes[:, None]]
    offs = (np.cumsum(sizes) - sizes).astype(np.uint32)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).cuda()
    dag = svdag_lib.MyGPUHashDAG(6, pool_bytes=1 << 30)
    table = dag.create_table(kind, [n // 16 + 1] * 9)
    handles = torch.empty(n, dtype=torch.int32, device="cuda")
    table.add(dev(flat), dev(offs), n, len(flat), handles)
    handles[::5] = -1  # a lookup that missed
    handles[3::7] = -2  # no item there
    out = torch.full((n * 10 + 3,), 77, dtype=torch.int32, device="cuda")
    table.read(handles, n, out[1:])
    torch.cuda.synchronize()
    want = words.copy()
    want[::5] = 0
    want[3::7] = 0
    got = out.cpu().numpy().view(np.uint32)
    assert np.array_equal(got[1:-2].reshape(n, 10), want)
    assert got[0] == 77 and got[-1] == 77 and got[-2] == 77
    dag.free()
