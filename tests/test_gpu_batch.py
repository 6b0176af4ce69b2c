"""Batched STQ on the GPU: many scenes through one launch sequence must give,
scene by scene, exactly the pairs of the oracle run on that scene alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def dev(arr, cuda):
    import torch

    return torch.from_numpy(np.ascontiguousarray(arr)).to(cuda)


@pytest.fixture(scope="module")
def scenes(stq, oracle):
    """24 cloth-pair scenes, box counts log-uniform in [1e3, 6e4], plus their
    oracle pair lists."""
    meshes = stq.batch_scenes(24, 1e3, 6e4, seed=5)
    want = []
    for m in meshes:
        b = oracle.construct_boxes(m.V0, m.V1, m.E, m.F, stq.AABB_DTYPE)
        want.append(oracle.broadphase(b))
    return meshes, want


def split_by_scene(pairs, box_off):
    s = np.searchsorted(box_off, pairs[:, 0], side="right") - 1
    s2 = np.searchsorted(box_off, pairs[:, 1], side="right") - 1
    assert np.array_equal(s, s2), "a pair crosses scenes"
    return s


def check_batch(oracle, raw, box_off, want, per_scene=None):
    got = oracle.canonical(raw)
    assert len(got) == len(raw), "duplicate pairs"
    sid = split_by_scene(got, box_off)
    for k, w in enumerate(want):
        local = got[sid == k] - box_off[k]
        assert np.array_equal(local, w), f"scene {k}"
        if per_scene is not None:
            assert per_scene[k] == len(w), f"scene {k} count"


def test_batch_build_matches_single_builds(ctx, stq, oracle, cuda, scenes):
    import torch

    meshes, _ = scenes
    V0, V1, E, F, vo, eo, fo = stq.concat_meshes(meshes)
    n = sum(m.num_boxes for m in meshes)
    out = torch.empty((n, 11), dtype=torch.int32, device=cuda)
    bo = ctx.batch_build_boxes(dev(V0, cuda), dev(V1, cuda), vo, dev(E, cuda), eo, dev(F, cuda), fo, out)
    assert bo[-1] == n
    got = out.cpu().numpy().view(stq.AABB_DTYPE).reshape(-1)
    for k, m in enumerate(meshes):
        want = oracle.construct_boxes(m.V0, m.V1, m.E, m.F, stq.AABB_DTYPE)
        part = got[bo[k]:bo[k + 1]].copy()
        assert np.array_equal(part["id"], np.arange(bo[k], bo[k + 1]))
        part["id"] -= bo[k]
        assert part.tobytes() == want.tobytes(), k


@pytest.mark.parametrize("shape", [1, 2])
@pytest.mark.parametrize("mixed_axes", [False, True])
@pytest.mark.parametrize("run_cap", [0, 3])
def test_batch_prepare_and_sweep(ctx, stq, oracle, cuda, scenes, mixed_axes, run_cap, shape):
    """Scene by scene against the oracle, with the per-scene pair counts
    (queue and flat shapes)."""
    import torch

    meshes, want = scenes
    ctx.set_option(stq.OPT_RUN_CAP, run_cap)
    ctx.set_option(stq.OPT_SWEEP_SHAPE, shape)
    V0, V1, E, F, vo, eo, fo = stq.concat_meshes(meshes)
    n = sum(m.num_boxes for m in meshes)
    boxes = torch.empty((n, 11), dtype=torch.int32, device=cuda)
    bo = ctx.batch_build_boxes(dev(V0, cuda), dev(V1, cuda), vo, dev(E, cuda), eo, dev(F, cuda), fo, boxes)
    axes = [(-1, 0, 1, 2)[k % 4] for k in range(len(meshes))] if mixed_axes else None
    ctx.batch_prepare(boxes, bo, axes=axes)
    cap = sum(len(w) for w in want) + 16
    pairs = torch.empty((cap, 2), dtype=torch.int32, device=cuda)
    r = ctx.sweep_prepared(pairs, cap)
    assert r.status == stq.STQ_OK and r.count == cap - 16
    per = ctx.batch_scene_pairs(len(meshes))
    check_batch(oracle, pairs[: r.count].cpu().numpy(), bo, want, per)


def test_batch_overflow_resume(ctx, stq, oracle, cuda, scenes):
    import torch

    meshes, want = scenes
    V0, V1, E, F, vo, eo, fo = stq.concat_meshes(meshes)
    n = sum(m.num_boxes for m in meshes)
    boxes = torch.empty((n, 11), dtype=torch.int32, device=cuda)
    bo = ctx.batch_build_boxes(dev(V0, cuda), dev(V1, cuda), vo, dev(E, cuda), eo, dev(F, cuda), fo, boxes)
    ctx.batch_prepare(boxes, bo)
    total = sum(len(w) for w in want)
    cap = total // 5 + 1
    pairs = torch.empty((cap, 2), dtype=torch.int32, device=cuda)
    start, parts = 0, []
    while start < ctx.prepared_length:
        r = ctx.sweep_prepared(pairs, cap, start=start)
        parts.append(pairs[: r.count].cpu().numpy().copy())
        start = r.next_start
    assert len(parts) >= 5
    check_batch(oracle, np.concatenate(parts), bo, want)


@pytest.mark.parametrize("graph", [1, 2])
@pytest.mark.parametrize("shape", [1, 2])
def test_batch_broadphase_fused(ctx, stq, oracle, cuda, scenes, graph, shape):
    import torch

    meshes, want = scenes
    ctx.set_option(stq.OPT_GRAPH, graph)
    ctx.set_option(stq.OPT_SWEEP_SHAPE, shape)
    V0, V1, E, F, vo, eo, fo = stq.concat_meshes(meshes)
    n = sum(m.num_boxes for m in meshes)
    bo = np.concatenate([[0], np.cumsum([m.num_boxes for m in meshes])])
    d = [dev(x, cuda) for x in (V0, V1, E, F)]
    cap = sum(len(w) for w in want) + 100
    pairs = torch.empty((cap, 2), dtype=torch.int32, device=cuda)
    for rep in range(3):  # the captured graph is replayed
        r, per = ctx.batch_broadphase(d[0], d[1], vo, d[2], eo, d[3], fo, pairs, cap)
        assert r.status == stq.STQ_OK
        check_batch(oracle, pairs[: r.count].cpu().numpy(), bo, want, per)
    # a different batch composition within the same capacities reuses the graph
    sub = meshes[::-1]
    V0b, V1b, Eb, Fb, vob, eob, fob = stq.concat_meshes(sub)
    for t, src in zip(d, (V0b, V1b, Eb, Fb)):
        t.copy_(dev(src, cuda))
    bob = np.concatenate([[0], np.cumsum([m.num_boxes for m in sub])])
    r, per = ctx.batch_broadphase(d[0], d[1], vob, d[2], eob, d[3], fob, pairs, cap)
    check_batch(oracle, pairs[: r.count].cpu().numpy(), bob, want[::-1], per)
    # too small a buffer reports overflow and the true total
    r, per = ctx.batch_broadphase(d[0], d[1], vob, d[2], eob, d[3], fob, pairs, 1000)
    assert r.status == stq.STQ_OVERFLOW and r.total == cap - 100 and r.count == 1000


def test_batch_with_empty_and_tiny_scenes(ctx, stq, oracle, cuda):
    import torch

    boxes = []
    for k, n in enumerate([0, 1, 2, 500, 0, 3000]):
        b = stq.random_boxes(n, seed=40 + k) if n else np.zeros(0, stq.AABB_DTYPE)
        if n:
            c = 0.5 * (b["min"] + b["max"])
            b["min"], b["max"] = c - 0.05, c + 0.05
        boxes.append(b)
    bo = np.concatenate([[0], np.cumsum([len(b) for b in boxes])]).astype(np.int64)
    allb = np.concatenate(boxes)
    allb["id"] = np.arange(len(allb))
    want = []
    for k, b in enumerate(boxes):
        bb = allb[bo[k]:bo[k + 1]].copy()
        want.append(oracle.broadphase(bb) - bo[k] if len(bb) else np.zeros((0, 2), np.int32))
    d = torch.from_numpy(allb.view(np.int32).reshape(-1, 11).copy()).to(cuda)
    ctx.batch_prepare(d, bo)
    cap = sum(len(w) for w in want) + 8
    pairs = torch.empty((cap, 2), dtype=torch.int32, device=cuda)
    r = ctx.sweep_prepared(pairs, cap)
    check_batch(oracle, pairs[: r.count].cpu().numpy(), bo, want, ctx.batch_scene_pairs(len(boxes)))


def test_batch_skewed_boxes_mixed_axes(ctx, stq, oracle, cuda):
    """Random boxes with 5% slivers stretched 200x, several scenes in one batch,
    the sweep axis fixed to x in half of them and chosen by variance in the
    others: each scene's pairs equal the oracle's on that scene alone."""
    import torch

    sizes = [30_000, 1, 12_000, 45_000, 0, 25_000]
    boxes = [stq.random_boxes(n, sliver_frac=0.05, seed=70 + k) if n else np.zeros(0, stq.AABB_DTYPE)
             for k, n in enumerate(sizes)]
    bo = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    allb = np.concatenate(boxes)
    allb["id"] = np.arange(len(allb))
    want = []
    for k in range(len(sizes)):
        bb = allb[bo[k]:bo[k + 1]].copy()
        want.append(oracle.broadphase(bb) - bo[k] if len(bb) else np.zeros((0, 2), np.int32))
    d = torch.from_numpy(allb.view(np.int32).reshape(-1, 11).copy()).to(cuda)
    axes = [0 if k % 2 == 0 else -1 for k in range(len(sizes))]
    ctx.batch_prepare(d, bo, axes=axes)
    cap = sum(len(w) for w in want) + 8
    pairs = torch.empty((cap, 2), dtype=torch.int32, device=cuda)
    r = ctx.sweep_prepared(pairs, cap)
    assert r.status == stq.STQ_OK
    check_batch(oracle, pairs[: r.count].cpu().numpy(), bo, want, ctx.batch_scene_pairs(len(sizes)))


@pytest.mark.parametrize("count", [256, 257, 2048, 2049, 5000])
def test_batches_of_many_small_scenes(ctx, stq, oracle, cuda, count):
    """More scenes (and tiles) than threads of the block that lays them out, empty ones
    and one of several tiles among them."""
    rng = np.random.default_rng(count)
    kinds = []
    for k in range(12):
        b = stq.random_boxes(5 * k, sliver_frac=0.0, seed=k) if k else np.zeros(0, stq.AABB_DTYPE)
        c = rng.uniform(0, 1, (len(b), 3)).astype(np.float32)
        b["min"], b["max"] = c, c + np.float32(0.3)
        kinds.append((b, oracle.broadphase(b) if k else np.zeros((0, 2), np.int32)))
    b = stq.random_boxes(3000, sliver_frac=0.0, seed=20)
    kinds.append((b, oracle.broadphase(b)))
    pick = rng.integers(0, 12, count)
    pick[[3, count - 2]] = 12
    bo = np.concatenate([[0], np.cumsum([len(kinds[k][0]) for k in pick])]).astype(np.int64)
    boxes = np.concatenate([kinds[k][0] for k in pick])
    boxes["id"] = np.arange(len(boxes))
    import torch

    want = [kinds[k][1] for k in pick]
    cap = sum(len(w) for w in want) + 16
    pairs = torch.empty((cap, 2), dtype=torch.int32, device=cuda)
    ctx.batch_prepare(dev(boxes.view(np.int32).reshape(-1, 11), cuda), bo)
    r = ctx.sweep_prepared(pairs, cap)
    assert r.status == stq.STQ_OK
    assert np.array_equal(ctx.batch_scene_pairs(count), [len(w) for w in want])
    all_want = np.concatenate([w + o for w, o in zip(want, bo[:-1])])
    assert np.array_equal(oracle.canonical(pairs[: r.count].cpu().numpy()), oracle.canonical(all_want))


def test_autotune_keeps_results_exact_and_caches(ctx, stq, oracle, cuda, scenes):
    import torch

    meshes, want = scenes
    V0, V1, E, F, vo, eo, fo = stq.concat_meshes(meshes)
    n = sum(m.num_boxes for m in meshes)
    boxes = torch.empty((n, 11), dtype=torch.int32, device=cuda)
    bo = ctx.batch_build_boxes(dev(V0, cuda), dev(V1, cuda), vo, dev(E, cuda), eo, dev(F, cuda), fo, boxes)
    cap = sum(len(w) for w in want) + 16
    pairs = torch.empty((cap, 2), dtype=torch.int32, device=cuda)
    ms, settings = ctx.autotune(boxes, bo, pairs, cap)
    assert ms > 0
    assert settings["shape"] in (stq.SHAPE_QUEUE, stq.SHAPE_FLAT)
    assert settings["lanes"] in (1, 4, 8, 16) and settings["queue"] in (16, 32, 64)
    assert settings["per_lane"] in (2, 4, 8) or settings["lanes"] > 1
    assert settings["queue"] >= 32 or settings["lanes"] > 1
    assert settings["run_cap"] in (512, 4096)
    assert settings["block"] in (128, 256, 512) and settings["radix_bits"] in (4, 8)
    assert settings["cell_scale"] in (1, 2, 4, 8)
    r = ctx.sweep_prepared(pairs, cap)
    check_batch(oracle, pairs[: r.count].cpu().numpy(), bo, want, ctx.batch_scene_pairs(len(meshes)))
    ms2, settings2 = ctx.autotune(boxes, bo, pairs, cap)  # same shape bucket: cached
    assert ms2 == 0 and settings2 == settings


@pytest.mark.parametrize("between", ["sort_pairs", "prepare"])
def test_batch_graph_follows_buffers_that_another_call_moved(stq, oracle, cuda, scenes, between):
    """A captured batch holds the context's buffers: a call between two batches
    that grows one of them (a sort of more pairs than the batch has replicas, a
    larger scene of one cell) makes the second batch capture again."""
    import torch

    meshes, want = scenes
    meshes, want = meshes[:4], want[:4]
    V0, V1, E, F, vo, eo, fo = stq.concat_meshes(meshes)
    d = [dev(x, cuda) for x in (V0, V1, E, F)]
    bo = np.concatenate([[0], np.cumsum([m.num_boxes for m in meshes])])
    cap = sum(len(w) for w in want) + 16
    pairs = torch.empty((cap, 2), dtype=torch.int32, device=cuda)
    with stq.Context(0, torch.cuda.current_stream(cuda).cuda_stream) as ctx:
        for rep in range(2):
            r, per = ctx.batch_broadphase(d[0], d[1], vo, d[2], eo, d[3], fo, pairs, cap)
            assert r.status == stq.STQ_OK
            check_batch(oracle, pairs[: r.count].cpu().numpy(), bo, want, per)
            if between == "sort_pairs":
                n = 40 * int(bo[-1])
                many = torch.randint(0, 1 << 20, (n, 2), dtype=torch.int32, device=cuda)
                ctx.sort_pairs(many, n)
            else:
                b = stq.random_boxes(3 * int(bo[-1]), seed=3)
                ctx.set_option(stq.OPT_CELLS, 1)
                ctx.prepare(dev(b.view(np.int32).reshape(-1, 11), cuda), len(b), 0)
                ctx.set_option(stq.OPT_CELLS, 0)


def test_scene_pairs_after_a_replayed_batch(stq, oracle, cuda, scenes):
    """A prepare between two batches that moves no buffer: the second batch replays the
    captured graph (no launch of its own), and the counts per scene are its own."""
    import torch

    meshes, want = scenes
    V0, V1, E, F, vo, eo, fo = stq.concat_meshes(meshes)
    d = [dev(x, cuda) for x in (V0, V1, E, F)]
    cap = sum(len(w) for w in want) + 16
    pairs = torch.empty((cap, 2), dtype=torch.int32, device=cuda)
    b = stq.random_boxes(64, seed=3)
    small = dev(b.view(np.int32).reshape(-1, 11), cuda)
    with stq.Context(0, torch.cuda.current_stream(cuda).cuda_stream) as ctx:
        for rep in range(3):
            before = ctx.launches
            r, per = ctx.batch_broadphase(d[0], d[1], vo, d[2], eo, d[3], fo, pairs, cap)
            assert r.status == stq.STQ_OK
            assert (ctx.launches == before) == (rep > 0)
            assert np.array_equal(per, [len(w) for w in want])
            assert np.array_equal(ctx.batch_scene_pairs(len(meshes)), per)
            ctx.prepare(small, len(b), 0)
            assert np.array_equal(ctx.batch_scene_pairs(1), [0])  # not swept yet


def test_batch_graph_outlives_growing_buffers_of_other_calls(ctx, stq, oracle, cuda, scenes):
    """Sorts of ever more pairs, an overflow's counts and a host call's copies are none of
    the captured batch's buffers: it is replayed (no launch of its own), not captured again."""
    import torch

    meshes, want = scenes
    V0, V1, E, F, vo, eo, fo = stq.concat_meshes(meshes)
    d = [dev(x, cuda) for x in (V0, V1, E, F)]
    cap = sum(len(w) for w in want) + 16
    pairs = torch.empty((cap, 2), dtype=torch.int32, device=cuda)
    few = stq.random_boxes(3000, seed=3)
    for rep in range(4):
        before = ctx.launches
        r, per = ctx.batch_broadphase(d[0], d[1], vo, d[2], eo, d[3], fo, pairs, cap)
        assert (ctx.launches == before) == (rep > 0)
        assert np.array_equal(per, [len(w) for w in want])
        if rep == 0:
            ctx.sweep_prepared(pairs, cap // 2)  # overflows
        elif rep == 1:
            many = torch.randint(0, 1 << 20, (cap, 2), dtype=torch.int32, device=cuda)
            ctx.sort_pairs(many, cap // 2)
            ctx.sort_pairs(many, cap)
        else:
            ctx.sweep_host(few, np.zeros((1 << 16 << rep, 2), np.int32), axis=0)


def test_batch_graph_follows_small_radii(ctx, stq, oracle, cuda, scenes):
    """Two inflation radii below 1e-9 are two graphs: the pairs of a scene scaled
    to 1e-9 depend on which of them was asked for."""
    import torch

    m = scenes[0][0]
    V0, V1 = m.V0 * 1e-9, m.V1 * 1e-9
    vo, eo, fo = ([0, len(x)] for x in (V0, m.E, m.F))
    d = [dev(x, cuda) for x in (V0, V1, m.E, m.F)]
    cap, counts = 64 * m.num_boxes, set()
    pairs = torch.empty((cap, 2), dtype=torch.int32, device=cuda)
    for r in (0.0, 2e-11, 0.0):
        want = oracle.broadphase(oracle.construct_boxes(V0, V1, m.E, m.F, stq.AABB_DTYPE, r))
        res, _ = ctx.batch_broadphase(d[0], d[1], vo, d[2], eo, d[3], fo, pairs, cap, inflation_radius=r)
        assert res.status == stq.STQ_OK
        assert np.array_equal(oracle.canonical(pairs[: res.count].cpu().numpy()), want)
        counts.add(len(want))
    assert len(counts) == 2


@pytest.mark.parametrize("filler", [0, 80_000, 640_000])  # tiles of 256, 1,024 and 4,096 boxes
def test_batch_build_at_tile_edges(ctx, stq, oracle, cuda, filler):
    import torch

    rng = np.random.default_rng(filler)
    sizes = [1, 31, 33, 0, 255, 256, 257, 1023, 1024, 1025, 4095, 4096, 4097, filler]
    vo = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    V0, V1 = rng.normal(size=(vo[-1], 3)), rng.normal(size=(vo[-1], 3))
    none = np.zeros(len(vo), np.int64)
    E, F = np.zeros((0, 2), np.int32), np.zeros((0, 3), np.int32)
    out = torch.full((int(vo[-1]) + 8, 11), -7, dtype=torch.int32, device=cuda)
    bo = ctx.batch_build_boxes(dev(V0, cuda), dev(V1, cuda), vo, dev(E, cuda), none, dev(F, cuda), none, out)
    assert np.array_equal(bo, vo)
    got = out.cpu().numpy()
    assert np.all(got[vo[-1] :] == -7)
    got = got[: vo[-1]].reshape(-1).view(stq.AABB_DTYPE)
    for a, b in zip(vo[:-1], vo[1:]):
        if a == b:
            continue
        want = oracle.construct_boxes(V0[a:b], V1[a:b], E, F, stq.AABB_DTYPE).copy()
        want["id"] += int(a)
        assert np.array_equal(got[a:b], want), (a, b)


def test_batch_build_at_edges_of_the_largest_tiles(ctx, stq, oracle, cuda):
    """As above in a batch above 1,245,184 boxes, whose tiles are of 4,096."""
    test_batch_build_at_tile_edges(ctx, stq, oracle, cuda, 1_240_000)
