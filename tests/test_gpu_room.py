"""One context over scenes that fit, outgrow and leave room in the buffers of the
scenes before: a sweep is queued whole where they may fit, and again where they
did not. Every call gives the oracle's pairs, and a bad box is refused from
either way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def scene(stq, n, side, seed):
    b = stq.random_boxes(n, sliver_frac=0.0, seed=seed)
    c = 0.5 * (b["min"] + b["max"])
    b["min"], b["max"] = c - np.float32(side / 2), c + np.float32(side / 2)
    return b


def dev(b, cuda):
    import torch

    return torch.from_numpy(b.view(np.int32).reshape(-1, 11).copy()).to(cuda)


@pytest.mark.parametrize("fused", [True, False])
def test_scenes_of_changing_size_and_density(ctx, stq, oracle, cuda, fused):
    import torch

    # boxes, side of a box: more replicas at the same count, more lists, more
    # digits of the replica sort, then small ones again; one scene twice
    steps = [(300, 0.05), (300, 0.05), (300, 0.3), (5000, 0.02), (5000, 0.09), (60_000, 0.01), (60_000, 0.02),
             (200_000, 0.004), (300, 0.05), (5000, 0.02)]
    for k, (n, side) in enumerate(steps):
        b = scene(stq, n, side, seed=50 + k)
        want = oracle.broadphase(b)
        pairs = torch.empty((len(want) + 16, 2), dtype=torch.int32, device=cuda)
        if fused:
            r = ctx.sweep(dev(b, cuda), n, pairs, len(want) + 16, axis=-1)
        else:
            ctx.prepare(dev(b, cuda), n, -1)
            assert np.array_equal(ctx.batch_scene_pairs(1), [0])  # not swept yet
            r = ctx.sweep_prepared(pairs, len(want) + 16)
        assert r.status == stq.STQ_OK and r.count == len(want) and r.next_start == ctx.prepared_length, k
        assert np.array_equal(oracle.canonical(pairs[: r.count].cpu().numpy()), want), k
        assert np.array_equal(ctx.batch_scene_pairs(1), [len(want)])


def test_bad_boxes_after_good_ones(ctx, stq, oracle, cuda):
    import torch

    b = scene(stq, 4000, 0.05, seed=7)
    want = oracle.broadphase(b)
    pairs = torch.empty((len(want) + 16, 2), dtype=torch.int32, device=cuda)
    bad = b.copy()
    bad["max"][17, 1] = np.nan
    for boxes, ok in ((b, True), (b, True), (bad, False), (b, True)):
        if ok:
            r = ctx.sweep(dev(boxes, cuda), len(b), pairs, len(want) + 16)
            assert r.count == len(want)
            assert np.array_equal(oracle.canonical(pairs[: r.count].cpu().numpy()), want)
        else:
            with pytest.raises(stq.STQError) as e:
                ctx.sweep(dev(boxes, cuda), len(b), pairs, len(want) + 16)
            assert e.value.status == stq.STQ_ERR_INVALID_INPUT and ctx.prepared_length == -1
    small = torch.empty((len(want) // 2, 2), dtype=torch.int32, device=cuda)
    r = ctx.sweep(dev(b, cuda), len(b), small, len(want) // 2)  # overflow from the whole call
    assert r.status == stq.STQ_OVERFLOW and r.total == len(want)
    got = [small[: r.count].cpu().numpy().copy()]
    while r.status == stq.STQ_OVERFLOW:
        r = ctx.sweep_prepared(small, len(want) // 2, start=r.next_start)
        got.append(small[: r.count].cpu().numpy().copy())
    assert np.array_equal(oracle.canonical(np.concatenate(got)), want)


def test_launches_follow_the_scene_not_the_buffers(stq, oracle, cuda):
    """A small scene on a context that has held a large one is launched like on one that
    has not, and a scene that outgrows the buffers is prepared twice, not three times."""
    import torch

    small, large = (300, scene(stq, 300, 0.05, seed=1)), (60_000, scene(stq, 60_000, 0.02, seed=2))
    pairs = torch.empty((1 << 20, 2), dtype=torch.int32, device=cuda)
    boxes = {n: dev(b, cuda) for n, b in (small, large)}
    want = {n: oracle.broadphase(b) for n, b in (small, large)}

    def launches(ctx, n):
        before = ctx.launches
        r = ctx.sweep(boxes[n], n, pairs, 1 << 20)
        assert np.array_equal(oracle.canonical(pairs[: r.count].cpu().numpy()), want[n])
        return ctx.launches - before

    stream = torch.cuda.current_stream(cuda).cuda_stream
    with stq.Context(0, stream) as a, stq.Context(0, stream) as b:
        first = launches(a, 300)
        again = launches(a, 300)
        first_large = launches(b, 60_000)
        assert launches(b, 300) == again  # no wait, the sort in one launch
        assert launches(a, 60_000) <= again + first_large
        assert first <= again


@pytest.mark.parametrize("field,axis", [(f, a) for f in ("min", "max") for a in range(3)])
@pytest.mark.parametrize("bits", [0x7FC00000, 0xFFC00000])  # NaN, and NaN with the sign set
def test_a_nan_of_either_sign_is_refused(ctx, stq, oracle, cuda, field, axis, bits):
    """In the first box, one in the middle and the last one of scenes in grids, by the whole
    sweep and by prepare; the scene without it before and after."""
    import torch

    n = 3000
    b = scene(stq, n, 0.04, seed=9)
    want = oracle.broadphase(b)
    good = dev(b, cuda)
    pairs = torch.empty((len(want) + 16, 2), dtype=torch.int32, device=cuda)
    for at in (0, n // 2, n - 1):
        bad = b.copy()
        bad[field].view(np.uint32)[at, axis] = bits
        bad = dev(bad, cuda)
        for cells in (0, 40):
            ctx.set_option(stq.OPT_CELLS, cells)
            for boxes in (good, bad, good):
                calls = (lambda: ctx.sweep(boxes, n, pairs, len(pairs), axis=-1),
                         lambda: ctx.batch_prepare(boxes, [0, 1, n], axis=0))
                for k, call in enumerate(calls):
                    if boxes is bad:
                        with pytest.raises(stq.STQError) as e:
                            call()
                        assert e.value.status == stq.STQ_ERR_INVALID_INPUT and ctx.prepared_length == -1
                    else:
                        r = call()
                        assert k or np.array_equal(oracle.canonical(pairs[: r.count].cpu().numpy()), want)


@pytest.mark.parametrize("left", [2500 << 20, 1500 << 20, 300 << 20])
def test_refused_allocations_leave_the_context_usable(stq, oracle, cuda, left):
    """The device's memory is held but for `left` bytes, so that the buffers of a large
    scene and a pair sort's are refused at different places. What fitted before fits
    after: the same small scene, against the oracle."""
    import torch

    b = scene(stq, 4000, 0.05, seed=7)
    want = oracle.broadphase(b)
    d, n = dev(b, cuda), len(b)
    pairs = torch.empty((len(want) + 16, 2), dtype=torch.int32, device=cuda)
    # 12 boxes across every cell of a 2,048 x 2,048 grid: 50 M replicas, 5 GB of buffers
    big = scene(stq, 12, 0.05, seed=8)
    big["min"], big["max"] = 0.0, 1.0
    big = dev(big, cuda)
    held = None

    def refused(call, *args):  # (an exception that is kept would keep the held memory)
        try:
            call(*args)
        except stq.STQError as e:
            return e.status
        return stq.STQ_OK

    with stq.Context(0, torch.cuda.current_stream(cuda).cuda_stream) as ctx:

        def check():
            r = ctx.sweep(d, n, pairs, len(want) + 16)
            assert r.status == stq.STQ_OK and r.count == len(want)
            ctx.sort_pairs(pairs, r.count)
            assert np.array_equal(pairs[: r.count].cpu().numpy(), oracle.canonical(want))

        check()
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info(cuda)[0]
        held = torch.empty(free - left, dtype=torch.uint8, device=cuda)
        try:
            ctx.set_option(stq.OPT_CELLS, 2048)
            assert refused(ctx.prepare, big, 12, 0) == stq.STQ_ERR_NO_MEMORY and ctx.prepared_length == -1
            assert refused(ctx.sweep_prepared, pairs, 16) == stq.STQ_ERR_NOT_PREPARED
            ctx.set_option(stq.OPT_CELLS, 0)
            check()
            # pairs (of the held memory, never read) whose second buffer fits, but not
            # the tables: half a byte per pair
            count = (torch.cuda.mem_get_info(cuda)[0] - (8 << 20)) // 8
            assert refused(ctx.sort_pairs, held, count) == stq.STQ_ERR_NO_MEMORY
            check()
        finally:
            del held
            torch.cuda.empty_cache()
