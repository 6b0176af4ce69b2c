"""The device sorts through stq_sort_pairs. Sizes at the edges of its kernels: one
block up to 4,096 and 8,192 pairs, buckets of about 2,560 (at most 4,096) pairs
above, segments of about 2^19 above 2^22. Ids that are few, wide, equal, or
uneven: neighbouring ids with more than 4,096 pairs take a large bucket, one first
id with more than 8,192 the radix sort, large groups of close pairs a bucket's
digits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def draw(rng, n, ids):
    if ids == "small":
        return rng.integers(0, 200, (n, 2), dtype=np.uint32)
    if ids == "wide":
        return rng.integers(0, 1 << 32, (n, 2), dtype=np.uint32)
    if ids == "equal":
        return np.full((n, 2), 7, np.uint32)
    if ids == "one_sided":
        p = rng.integers(0, 70_000, (n, 2), dtype=np.uint32)
        p[:, 0] = 5
        return p
    if ids == "groups":  # first ids of about 150 pairs each
        p = rng.integers(0, 1 << 22, (n, 2), dtype=np.uint32)
        p[:, 0] = rng.integers(0, max(n // 150, 1), n)
        return p
    if ids == "clumps":  # of about 600, in two narrow ranges of second ids
        p = rng.integers(0, 250, (n, 2), dtype=np.uint32)
        p[:, 1] += rng.integers(0, 2, n, dtype=np.uint32) << 30
        p[:, 0] = rng.integers(0, max(n // 600, 1), n)
        return p
    if ids == "dense":  # 6,000 pairs of eight neighbouring ids
        p = rng.integers(0, max(n // 4, 2), (n, 2), dtype=np.uint32)
        at = rng.choice(n, min(n, 6000), replace=False)
        p[at, 0] = n // 9 + rng.integers(0, 8, len(at))
        return p
    if ids == "hub":  # a scene in which one box meets 1 in 50
        p = rng.integers(0, max(n // 4, 2), (n, 2), dtype=np.uint32)
        p[:: 50, 0] = n // 9
        return p
    p = rng.integers(0, max(n // 4, 2), (n, 2), dtype=np.uint32)  # "scene": 4 pairs per box
    return np.sort(p, axis=1)


def check(ctx, cuda, p):
    import torch

    n = len(p)
    want = p[np.lexsort((p[:, 1], p[:, 0]))]
    buf = torch.full((n + 64, 2), -7, dtype=torch.int32, device=cuda)
    buf[:n] = torch.from_numpy(p.view(np.int32)).to(cuda)
    ctx.sort_pairs(buf, n)
    got = buf.cpu().numpy()
    assert np.array_equal(got[:n].view(np.uint32), want)
    assert np.all(got[n:] == -7)  # nothing written past the end


@pytest.mark.parametrize("n", [2, 33, 1023, 4095, 4096, 4097, 8191, 8192, 8193, 10241, 100_003, 933_889, 2_000_003])
@pytest.mark.parametrize("ids", ["small", "one_sided", "wide", "equal", "groups", "clumps", "dense", "hub", "scene"])
def test_sort_pairs_sizes_and_ids(ctx, cuda, n, ids):
    check(ctx, cuda, draw(np.random.default_rng(n), n, ids))


@pytest.mark.parametrize("n", [(1 << 22) - 1, (1 << 22) + 1, 9_500_000])
@pytest.mark.parametrize("ids", ["small", "wide", "groups", "clumps", "dense", "hub", "scene"])
def test_sort_pairs_segments(ctx, cuda, n, ids):
    check(ctx, cuda, draw(np.random.default_rng(n), n, ids))


def test_sort_pairs_ids_that_grow_and_shrink(ctx, cuda):
    """The bins' width follows the ids of earlier sorts: ids above it, and far
    below it, sort the same."""
    rng = np.random.default_rng(3)
    for hi in (1000, 1 << 30, 50, 70_000, 1 << 20, 9):
        check(ctx, cuda, rng.integers(0, hi, (60_000, 2), dtype=np.uint32))


@pytest.mark.parametrize("n", [5, 5000, 20_001])
def test_sort_pairs_on_a_four_byte_boundary(ctx, cuda, n):
    """A pair is two 32-bit ids: any 4-byte boundary is taken."""
    import torch

    p = draw(np.random.default_rng(n), n, "scene")
    flat = torch.full((2 * n + 3,), -7, dtype=torch.int32, device=cuda)
    flat[1 : 2 * n + 1] = torch.from_numpy(p.view(np.int32).reshape(-1)).to(cuda)
    ctx.sort_pairs(flat[1:], n)
    got = flat.cpu().numpy()
    assert np.array_equal(got[1 : 2 * n + 1].view(np.uint32).reshape(n, 2), p[np.lexsort((p[:, 1], p[:, 0]))])
    assert got[0] == -7 and np.all(got[2 * n + 1 :] == -7)
