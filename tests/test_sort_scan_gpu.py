"""The spatial sort's offset scan: one block of chunks, one batch of blocks
(the top scan in one group of threads) and more (four groups).  With one
feature the cells are 2^16 intervals of the range, so the sorted points ascend
up to one cell, and points of equal value keep their order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CHUNK, BATCH = 4096, 16  # points of a chunk (d = 1), chunks of a scan block at least


@pytest.mark.parametrize("n", [1, CHUNK, CHUNK + 1, CHUNK * BATCH, CHUNK * BATCH + 1, CHUNK * BATCH * BATCH - 3,
                               CHUNK * BATCH * BATCH, CHUNK * BATCH * BATCH + 1, 3 * CHUNK * BATCH * BATCH + 77])
def test_scan_blocks(ckm, cuda, n):
    import torch
    g = torch.Generator(device=cuda).manual_seed(n)
    x = torch.randint(0, 50000, (n,), generator=g, device=cuda).float()
    x[0] = 0.0
    x[-1] = 25000.0
    out, perm = ckm.spatial_sort(x, n, 1)
    p = perm.cpu().numpy().view(np.uint32).astype(np.int64)
    v = out.cpu().numpy()
    assert np.array_equal(np.sort(p), np.arange(n))
    assert np.array_equal(v, x.cpu().numpy()[p])
    # cells are narrower than the distance of two values
    assert np.all(np.diff(v) >= 0)
    same = np.diff(v) == 0
    assert np.all(np.diff(p)[same] > 0)
    back = torch.full((n,), -1, dtype=torch.int32, device=cuda)
    ckm.unpermute(perm, torch.arange(n, dtype=torch.int32, device=cuda), back, n)
    assert np.array_equal(back.cpu().numpy()[p], np.arange(n))
