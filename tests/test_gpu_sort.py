"""The device radix sort through stq_sort_pairs: sizes at the edges of its
kernels (one block up to 1,024 / 4,096 / 8,192 pairs, tiles of 2,048 and 6,144
pairs above), ids that use one digit, all four, or none."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 33, 1023, 1024, 1025, 4095, 4097, 8191, 8192, 8193, 10241, 100_003, 933_887, 933_889,
                               2_000_003])
@pytest.mark.parametrize("ids", ["small", "one_sided", "wide", "equal"])
def test_sort_pairs_sizes_and_ids(ctx, cuda, n, ids):
    import torch

    rng = np.random.default_rng(n)
    hi = {"small": 200, "one_sided": 70_000, "wide": 1 << 32, "equal": 1}[ids]
    p = rng.integers(0, hi, (n, 2), dtype=np.uint32)
    if ids == "one_sided":
        p[:, 0] = 5
    want = p[np.lexsort((p[:, 1], p[:, 0]))]
    buf = torch.full((n + 64, 2), -7, dtype=torch.int32, device=cuda)
    buf[:n] = torch.from_numpy(p.view(np.int32)).to(cuda)
    ctx.sort_pairs(buf, n)
    got = buf.cpu().numpy()
    assert np.array_equal(got[:n].view(np.uint32), want)
    assert np.all(got[n:] == -7)  # nothing written past the end
