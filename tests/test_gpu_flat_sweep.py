"""The flat sweep's forms: windows where every code passes (32 x 32 candidates per
step, more than a queue round), runs cut by the cap, a mix of dense and sparse
starts, and overflow counts from the same kernel; all against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def dense_boxes(stq, n, seed, spread):
    """n boxes of which most overlap: side 1, centres within `spread`."""
    b = stq.random_boxes(n, sliver_frac=0.0, seed=seed)
    rng = np.random.default_rng(seed)
    c = rng.uniform(0, spread, (n, 3)).astype(np.float32)
    b["min"], b["max"] = c - np.float32(0.5), c + np.float32(0.5)
    # unrelated ids, so that few pairs share a vertex
    b["vertex_ids"][:, 0] = np.arange(n)
    b["vertex_ids"][:, 1] = np.where(b["vertex_ids"][:, 1] >= 0, n + np.arange(n), -np.arange(n) - 1)
    b["vertex_ids"][:, 2] = np.where(b["vertex_ids"][:, 2] >= 0, 2 * n + np.arange(n), -np.arange(n) - 1)
    return b


@pytest.mark.parametrize("n", [2, 31, 32, 33, 64, 65, 300, 1100, 2500])
@pytest.mark.parametrize("spread", [0.0, 1.0, 40.0])
@pytest.mark.parametrize("run_cap", [0, 40])
def test_dense_windows_vs_oracle(ctx, stq, oracle, cuda, n, spread, run_cap):
    import torch

    b = dense_boxes(stq, n, 5 + n, spread)
    want = oracle.broadphase(b)
    d = torch.from_numpy(b.view(np.int32).reshape(-1, 11).copy()).to(cuda)
    ctx.set_option(stq.OPT_RUN_CAP, run_cap)
    cap = len(want) + 16
    pairs = torch.empty((cap, 2), dtype=torch.int32, device=cuda)
    for axis in (0, -1):
        r = ctx.sweep(d, n, pairs, cap, axis=axis)
        assert r.status == stq.STQ_OK and r.count == len(want)
        assert np.array_equal(oracle.canonical(pairs[: r.count].cpu().numpy()), want)
    if len(want) < 64:
        return
    most = 1 + max(len(want) // 5, 4 * n)  # one start box has at most n pairs
    start, parts = 0, []
    while start < ctx.prepared_length:
        r = ctx.sweep_prepared(pairs, min(most, cap), start=start)
        parts.append(pairs[: r.count].cpu().numpy().copy())
        start = r.next_start
    got = np.concatenate(parts)
    assert len(got) == len(want) and np.array_equal(oracle.canonical(got), want)


@pytest.mark.parametrize("n", [255, 256, 257, 77_823, 77_824, 77_825, 622_592, 622_593])
def test_tile_edges_vs_oracle(ctx, stq, oracle, cuda, n):
    """Tiles of 256 boxes up to 77,824 boxes, of 1,024 up to 622,592, of 2,048 above;
    the last one full, one short of it, or of one box."""
    import torch

    b = stq.random_boxes(n, seed=n)
    want = oracle.broadphase(b)
    d = torch.from_numpy(b.view(np.int32).reshape(-1, 11).copy()).to(cuda)
    cap = len(want) + 16
    pairs = torch.empty((cap, 2), dtype=torch.int32, device=cuda)
    r = ctx.sweep(d, n, pairs, cap, axis=-1)
    assert r.status == stq.STQ_OK and r.count == len(want)
    assert np.array_equal(oracle.canonical(pairs[: r.count].cpu().numpy()), want)


@pytest.mark.parametrize("n", [1_245_184, 1_245_185])
def test_large_tile_edges_vs_oracle(ctx, stq, oracle, cuda, n):
    """Tiles of 2,048 boxes up to 1,245,184 boxes, of 4,096 above."""
    import torch

    b = stq.random_boxes(n, sliver_frac=0.0, seed=n)
    want = oracle.broadphase(b)
    d = torch.from_numpy(b.view(np.int32).reshape(-1, 11).copy()).to(cuda)
    cap = len(want) + 16
    pairs = torch.empty((cap, 2), dtype=torch.int32, device=cuda)
    for _ in range(2):
        r = ctx.sweep(d, n, pairs, cap, axis=-1)
        assert r.status == stq.STQ_OK and r.count == len(want)
        assert np.array_equal(oracle.canonical(pairs[: r.count].cpu().numpy()), want)


@pytest.mark.parametrize("shape", [1, 2])
@pytest.mark.parametrize("run_cap", [0, 40])
def test_windows_after_an_overflow(ctx, stq, oracle, cuda, shape, run_cap):
    """Windows after the first that overflowed count while they emit (flat shape):
    windows that overflow, the last one with room to spare, one that fits exactly,
    and one a pair short."""
    import torch

    n = 1500
    b = dense_boxes(stq, n, 3, 6.0)
    want = oracle.broadphase(b)
    d = torch.from_numpy(b.view(np.int32).reshape(-1, 11).copy()).to(cuda)
    ctx.set_option(stq.OPT_SWEEP_SHAPE, shape)
    ctx.set_option(stq.OPT_RUN_CAP, run_cap)
    pairs = torch.empty((len(want) + 16, 2), dtype=torch.int32, device=cuda)
    ctx.prepare(d, n, 0)
    for most in (len(want) // 3, len(want) // 7 + n):
        start, parts = 0, []
        while start < ctx.prepared_length:
            r = ctx.sweep_prepared(pairs, most, start=start)
            assert r.count <= most and r.next_start > start
            assert (r.status == stq.STQ_OK) == (r.next_start == ctx.prepared_length)
            parts.append(pairs[: r.count].cpu().numpy().copy())
            start = r.next_start
        got = np.concatenate(parts)
        assert len(got) == len(want) and np.array_equal(oracle.canonical(got), want)
    r = ctx.sweep_prepared(pairs, len(want))  # fits exactly
    assert r.status == stq.STQ_OK and r.count == r.total == len(want)
    assert np.array_equal(oracle.canonical(pairs[: r.count].cpu().numpy()), want)
    r = ctx.sweep_prepared(pairs, len(want) - 1)
    assert r.status == stq.STQ_OVERFLOW and r.total == len(want) and r.count < len(want)


def overlaps_on_x(b, axis):
    """Pairs that overlap on the axis, of two edges or of a vertex and a face."""
    kind = (b["vertex_ids"][:, 1] >= 0).astype(int) + (b["vertex_ids"][:, 2] >= 0)
    lo, hi = b["min"][:, axis], b["max"][:, axis]
    order = [np.argsort(lo[kind == k], kind="stable") for k in range(3)]
    v, e, f = ((lo[kind == k][order[k]], hi[kind == k][order[k]]) for k in range(3))
    to = lambda x, bound, side="right": np.searchsorted(x[0], bound, side)  # noqa: E731
    edges = (to(e, e[1]) - np.arange(len(e[0])) - 1).sum()
    return int(edges + (to(f, v[1]) - to(f, v[0], "left")).sum() + (to(v, f[1]) - to(v, f[0])).sum())


@pytest.mark.parametrize("spread", ["even", "far", "far both", "clusters"])
@pytest.mark.parametrize("axis", [0, 2])
def test_candidates_of_one_long_list(ctx, stq, oracle, cuda, spread, axis):
    """However the boxes lie on the sweep axis, one list's candidates are those that
    overlap on it: a box far away or gaps do not put boxes on one code."""
    import torch

    n = 60_000
    b = stq.random_boxes(n, sliver_frac=0.0, seed=4)
    rng = np.random.default_rng(4)
    lo = rng.uniform(0, 1, (n, 3)).astype(np.float32)
    if spread == "clusters":
        lo[:, axis] = (rng.integers(0, 150, n) + 1e-3 * lo[:, axis]) / 150
    if spread in ("far", "far both"):
        lo[17, axis] = 1e4
    if spread == "far both":
        lo[18, axis] = -1e5
    b["min"], b["max"] = lo, lo + np.float32(1e-6 if spread == "clusters" else 1e-3)
    want, real = oracle.broadphase(b), overlaps_on_x(b, axis)
    pairs = torch.empty((len(want) + 16, 2), dtype=torch.int32, device=cuda)
    ctx.set_option(stq.OPT_CELLS, 1)
    d = torch.from_numpy(b.view(np.int32).reshape(-1, 11).copy()).to(cuda)
    for _ in range(2):
        r = ctx.sweep(d, n, pairs, len(want) + 16, axis=axis)
        assert r.count == len(want)
        assert np.array_equal(oracle.canonical(pairs[: r.count].cpu().numpy()), want)
        assert real <= ctx.candidates <= 1.01 * real + 100


@pytest.mark.parametrize("n", [12_287, 12_288, 12_289, 40_000])
def test_long_list_keys_vs_oracle(ctx, stq, oracle, cuda, n):
    """Either side of the line from which a list's keys are those of the minima (4,096
    boxes per list, three lists in a scene): negative and equal minima, both zeros,
    infinite bounds, and boxes inverted on the sweep axis."""
    import torch

    b = dense_boxes(stq, n, n, 400.0)
    centre = 0.5 * (b["min"] + b["max"]) - np.float32(200)
    centre[:, 1:] /= 40
    b["min"], b["max"] = centre - np.float32(0.5), centre + np.float32(0.5)
    for side in ("min", "max"):
        b[side][: n // 2, 0] = np.round(b[side][: n // 2, 0])  # (-0 among them)
    b["max"][5, 0], b["min"][6, 0], b["max"][7, 1], b["min"][8, 2] = np.inf, -np.inf, np.inf, -np.inf
    b["min"][9, 0], b["max"][9, 0] = 1.25, -3.75
    b["min"][10, 0], b["max"][10, 0] = 150.125, -np.inf
    want = oracle.broadphase(b)
    d = torch.from_numpy(b.view(np.int32).reshape(-1, 11).copy()).to(cuda)
    pairs = torch.empty((len(want) + 16, 2), dtype=torch.int32, device=cuda)
    ctx.set_option(stq.OPT_CELLS, 1)
    for _ in range(2):
        r = ctx.sweep(d, n, pairs, len(want) + 16, axis=0)
        assert r.count == len(want)
        assert np.array_equal(oracle.canonical(pairs[: r.count].cpu().numpy()), want)
    ctx.batch_prepare(d, [0, 0, n // 2, n], axis=0)  # lists half as long, an empty scene between
    r = ctx.sweep_prepared(pairs, len(want) + 16)
    halves = [oracle.broadphase(b[: n // 2]), oracle.broadphase(b[n // 2 :])]
    want = np.concatenate([h for h in halves if len(h)])
    assert np.array_equal(oracle.canonical(pairs[: r.count].cpu().numpy()), oracle.canonical(want))


def test_runs_of_tens_of_millions(ctx, stq, cuda):
    """2,500 boxes along the whole axis above 70 M points on it: one list, in which 32 of
    the long runs together have more candidates than 31 bits count. The long boxes all
    meet each other and no point; a point meets none."""
    import torch

    n, long = 70_000_000, 2500
    boxes = torch.zeros((n + long, 11), dtype=torch.int32, device=cuda)
    i = torch.arange(n + long, dtype=torch.int32, device=cuda)
    boxes[:, 0] = i
    x = (i[:n] + 0x3F800000).view(torch.float32)  # 70 M floats from 1 on
    f = boxes.view(torch.float32)
    f[:n, 1] = x
    f[:n, 4] = x
    f[n:, 1] = 0.5
    f[n:, 4] = float(x[-1])
    f[n:, [2, 3, 5, 6]] = 1.0  # y and z of the long boxes
    boxes[:, 7], boxes[:, 8], boxes[:, 9] = 2 * i, 2 * i + 1, -2 * i - 1  # edges without a common vertex
    ctx.set_option(stq.OPT_CELLS, 1)
    want = long * (long - 1) // 2
    pairs = torch.empty((want + 16, 2), dtype=torch.int32, device=cuda)
    r = ctx.sweep(boxes, n + long, pairs, want + 16, axis=0)
    assert r.status == stq.STQ_OK and r.count == want
    ctx.sort_pairs(pairs, want)
    a, b = torch.triu_indices(long, long, 1, device=cuda).to(torch.int32)
    assert torch.equal(pairs[:want, 0], a + n) and torch.equal(pairs[:want, 1], b + n)
