"""The work that programs have this library do, as cases that can be timed.

Each case is one pass through the public entry points (the Python binding of
include/stq_abi.h), from the smallest scene, where latency and launches count,
to the largest:

  step    one simulation step on a device mesh: swept boxes, sweep, and the
          pairs put in order (the sweep writes them in no particular order; a
          program whose steps must repeat bit for bit sorts them)
  resume  the same with a pair buffer that holds only part of the pairs: sweep
          until it is full, resume from the cursor, until all start boxes are done
  batch   many meshes through the fused, graph-captured batched call
  boxes   many scenes of ready-made boxes: batched prepare, sweep, counts per scene
  static  the allocation-free sweep of a small scene
  host    host boxes in, host pairs out (the caller sorts them on the host)
  serve   a burst of time-stepped requests through the server, until all are done

Pairs come back as the caller's whole buffer and the number found: the buffers
start at zero, and nothing is written past that number. Every output is a whole
number (pair ids, counts, checksums) or the bytes of a box, so there is nothing
to state in higher precision.
"""
import ctypes
import importlib
import math
import random

import numpy as np
import torch

stq = importlib.import_module("broadphase-gpu_gb300").stq

DEVICE = "cuda:0"
PAIRS_PER_BOX = 24  # pair buffers: above the densest scene of the ranges below


def listed():
    return [
        # a rigid part or a small garment in a real-time loop that may not allocate
        dict(name="static_small", kind="static", scene="cloth", g=9, z_offset=0.01, motion=0.6, axis=0),
        # the largest scene of the allocation-free call: boxes of mixed size with slivers
        dict(name="static_65k", kind="static", scene="random", boxes=65536, axis=1),
        # a small interactive scene, library defaults
        dict(name="step_cloth_2k", kind="step", scene="cloth", g=13, z_offset=0.02, motion=0.3, axis=-1,
             inflation=0.0, cell_scale=0),
        # an ordinary garment step with a contact margin and the axis known beforehand
        dict(name="step_cloth_53k", kind="step", scene="cloth", g=67, z_offset=0.01, motion=0.5, axis=0,
             inflation=1e-3, cell_scale=0),
        # the cloth-pair benchmark scene (two sheets of 200 x 200 vertices)
        dict(name="step_cloth_477k", kind="step", scene="cloth", g=200, z_offset=0.01, motion=0.6, axis=-1,
             inflation=0.0, cell_scale=0),
        # the large benchmark scene (16 crumpled sheets of 250 x 250) at the tuned cell size
        dict(name="step_crumpled_6m", kind="step", scene="crumpled", sheets=16, g=250, axis=-1, inflation=0.0,
             cell_scale=4),
        # a pair buffer for a third of the pairs: narrow phase after each part
        dict(name="resume_crumpled_684k", kind="resume", scene="crumpled", sheets=8, g=120, axis=-1,
             inflation=0.0, cell_scale=0, window=1.2),
        # many small scenes at once (learning environments, parameter sweeps)
        dict(name="batch_16_small", kind="batch", scenes=16, lo=1e3, hi=2e4, cell_scale=0, per_lane=0),
        # the batched benchmark: 256 scenes, tuned
        dict(name="batch_256", kind="batch", scenes=256, lo=1e3, hi=2e5, cell_scale=4, per_lane=2),
        # scenes of unrelated boxes with slivers, x and the largest-variance axis in turn
        dict(name="boxes_16x500k", kind="boxes", scenes=16, per=500_000, cell_scale=8),
        # boxes that live on the host, pairs wanted there
        dict(name="host_200k", kind="host", boxes=200_001, axis=-1),
        # a burst of requests of very different sizes, 1 to 20 timesteps each
        dict(name="serve_24", kind="serve", requests=24, lo=1e4, hi=1e6, max_steps=20),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _cloth(rng, g):
    return dict(scene="cloth", g=g, z_offset=round(rng.uniform(0.002, 0.05), 4), motion=round(rng.uniform(0.2, 0.9), 3))


def draw(rng: random.Random):
    kind = rng.choice(["step", "step", "step", "resume", "batch", "batch", "boxes", "static", "host", "serve"])
    if kind in ("step", "resume"):
        c = dict(kind=kind, axis=rng.choice([-1, -1, 0, 1, 2]), inflation=rng.choice([0.0, 0.0, 2.5e-4]),
                 cell_scale=rng.choice([0, 0, 4]))
        if rng.random() < 0.5:
            c.update(_cloth(rng, int(_log(rng, 9, 230))))
        else:
            c.update(scene="crumpled", sheets=rng.randint(2, 14), g=int(_log(rng, 20, 230)))
        if kind == "resume":
            c["window"] = round(_log(rng, 0.5, 4.0), 3)
        return c
    if kind == "batch":
        hi = _log(rng, 5e3, 2e5)
        return dict(kind=kind, scenes=int(_log(rng, 2, 200)), lo=1e3, hi=round(hi), cell_scale=rng.choice([0, 4]),
                    per_lane=rng.choice([0, 2]))
    if kind == "boxes":
        return dict(kind=kind, scenes=int(_log(rng, 1, 14)), per=int(_log(rng, 2e4, 5e5)), cell_scale=rng.choice([0, 4, 8]))
    if kind == "static":
        if rng.random() < 0.5:
            return dict(kind=kind, scene="random", boxes=int(_log(rng, 2e4, 65536)), axis=rng.randint(0, 2))
        return dict(kind=kind, axis=rng.randint(0, 2), **_cloth(rng, int(_log(rng, 5, 70))))
    if kind == "host":
        return dict(kind=kind, boxes=int(_log(rng, 2e4, 4e5)), axis=rng.choice([-1, 0, 2]))
    hi = _log(rng, 3e4, 6e5)
    return dict(kind="serve", requests=int(_log(rng, 1, 20)), lo=round(hi / 30), hi=round(hi), max_steps=rng.randint(2, 16))


# ---- scenes -----------------------------------------------------------------------

def _mesh(c, seed):
    if c["scene"] == "cloth":  # motion: its standard deviation in vertex spacings
        return stq.cloth_pair(g=c["g"], z_offset=c["z_offset"], sigma=c["motion"] / (c["g"] - 1), seed=seed)
    return stq.crumpled_sheets(sheets=c["sheets"], g=c["g"], seed=seed)


def _boxes(n, seed):
    return stq.random_boxes(n, sliver_frac=0.05, seed=seed)


def _device(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEVICE)


def _box_tensor(boxes):
    return _device(boxes.view(np.int32).reshape(-1, 11))


def _pair_buffer(n, per_box=PAIRS_PER_BOX):
    return torch.zeros((per_box * n + 1024, 2), dtype=torch.int32, device=DEVICE)


def _context(c):
    ctx = stq.Context(0, torch.cuda.current_stream().cuda_stream)
    if c.get("cell_scale"):
        ctx.set_option(stq.OPT_CELL_SCALE, c["cell_scale"])
    if c.get("per_lane"):
        ctx.set_option(stq.OPT_PER_LANE, c["per_lane"])
    return ctx


def _cloth_scenes(count, lo, hi, seed):
    """Cloth pairs with box counts spread evenly over the logarithm of [lo, hi], in an
    order that the case alone fixes; offsets, motions and positions come from the seed."""
    sizes = [lo * (hi / lo) ** ((k + 0.5) / count) for k in range(count)]
    random.Random(count).shuffle(sizes)
    rng = np.random.default_rng(seed)
    return [stq.cloth_pair(g=stq.cloth_pair_grid_for(int(n)), z_offset=float(rng.uniform(0.002, 0.05)),
                           sigma=float(rng.uniform(0.001, 0.01)), seed=int(rng.integers(1 << 40))) for n in sizes]


def _requests(c, seed):
    """(mesh, steps, seed of its motion): the steps are spread over 1 .. max_steps."""
    meshes = _cloth_scenes(c["requests"], c["lo"], c["hi"], seed)
    last = max(1, c["requests"] - 1)
    return [(m, 1 + k * (c["max_steps"] - 1) // last, seed * 1000 + k) for k, m in enumerate(meshes)]


def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    s = dict(case=c)
    if kind in ("step", "resume"):
        m = _mesh(c, seed)
        s.update(ctx=_context(c), n=m.num_boxes, V0=_device(m.V0), V1=_device(m.V1), E=_device(m.E), F=_device(m.F),
                 boxes=torch.empty((m.num_boxes, 11), dtype=torch.int32, device=DEVICE), pairs=_pair_buffer(m.num_boxes))
    elif kind == "batch":
        meshes = _cloth_scenes(c["scenes"], c["lo"], c["hi"], seed)
        V0, V1, E, F, vo, eo, fo = stq.concat_meshes(meshes)
        # the pairs are sorted through a context of their own: the batched call's
        # captured graph keeps its context's buffers
        s.update(ctx=_context(c), sorter=_context({}), V0=_device(V0), V1=_device(V1), E=_device(E), F=_device(F),
                 vo=vo, eo=eo, fo=fo, pairs=_pair_buffer(sum(m.num_boxes for m in meshes)))
    elif kind == "boxes":
        scenes = [_boxes(c["per"], seed * 1000 + k) for k in range(c["scenes"])]
        every = np.concatenate(scenes)
        every["id"] = np.arange(len(every), dtype=np.int32)
        s.update(ctx=_context(c), boxes=_box_tensor(every), off=np.arange(c["scenes"] + 1, dtype=np.int64) * c["per"],
                 axes=[stq.AXIS_X if k % 2 == 0 else stq.AXIS_AUTO for k in range(c["scenes"])],
                 pairs=_pair_buffer(len(every), 1))
    elif kind == "static":
        ctx = _context(c)
        if c["scene"] == "random":
            n, boxes = c["boxes"], _box_tensor(_boxes(c["boxes"], seed))
        else:
            m = _mesh(c, seed)
            n = m.num_boxes
            boxes = torch.empty((n, 11), dtype=torch.int32, device=DEVICE)
            ctx.build_boxes(_device(m.V0), _device(m.V1), _device(m.E), _device(m.F), boxes)
        s.update(ctx=ctx, n=n, boxes=boxes, pairs=_pair_buffer(n), lib=stq.load_library(),
                 stream=torch.cuda.current_stream().cuda_stream)
    elif kind == "host":
        boxes = _boxes(c["boxes"], seed)
        pinned = torch.empty((c["boxes"], 11), dtype=torch.int32, pin_memory=True)
        pinned.copy_(torch.from_numpy(boxes.view(np.int32).reshape(-1, 11)))
        pairs = torch.zeros((c["boxes"] + 1024, 2), dtype=torch.int32, pin_memory=True)
        s.update(ctx=_context(c), held=(pinned, pairs), boxes=pinned.numpy().view(stq.AABB_DTYPE).reshape(-1),
                 pairs=pairs.numpy())
    else:
        reqs = _requests(c, seed)
        boxes = sum(m.num_boxes for m, _, _ in reqs)
        s.update(server=stq.Server(0, None, budget_bytes=80 << 30, max_boxes=max(boxes, 1 << 16),
                                   max_scenes=max(32, c["requests"])), requests=reqs)
    return s


# ---- passes -----------------------------------------------------------------------

def _all(r):
    if r.status != stq.STQ_OK:
        raise RuntimeError("the pair buffer is too small: %r" % (r,))
    return r.count


def run(state):
    s, c = state, state["case"]
    kind = c["kind"]
    if kind == "step":
        ctx, pairs = s["ctx"], s["pairs"]
        ctx.build_boxes(s["V0"], s["V1"], s["E"], s["F"], s["boxes"], c["inflation"])
        count = _all(ctx.sweep(s["boxes"], s["n"], pairs, pairs.shape[0], axis=c["axis"]))
        ctx.sort_pairs(pairs, count)
        return dict(boxes=s["boxes"], count=count, pairs=pairs)
    if kind == "resume":
        ctx, pairs = s["ctx"], s["pairs"]
        window = int(c["window"] * s["n"])
        ctx.build_boxes(s["V0"], s["V1"], s["E"], s["F"], s["boxes"], c["inflation"])
        ctx.prepare(s["boxes"], s["n"], c["axis"])
        count = start = 0
        while True:
            r = ctx.sweep_prepared(pairs[count:], min(window, pairs.shape[0] - count), start)
            count, start = count + r.count, r.next_start
            if r.status == stq.STQ_OK:
                break
        ctx.sort_pairs(pairs, count)
        return dict(boxes=s["boxes"], count=count, pairs=pairs)
    if kind == "batch":
        ctx, pairs = s["ctx"], s["pairs"]
        r, per_scene = ctx.batch_broadphase(s["V0"], s["V1"], s["vo"], s["E"], s["eo"], s["F"], s["fo"], pairs,
                                            pairs.shape[0])
        s["sorter"].sort_pairs(pairs, _all(r))
        return dict(per_scene=per_scene, count=r.count, pairs=pairs)
    if kind == "boxes":
        ctx, pairs = s["ctx"], s["pairs"]
        ctx.batch_prepare(s["boxes"], s["off"], axes=s["axes"])
        count = _all(ctx.sweep_prepared(pairs, pairs.shape[0]))
        per_scene = ctx.batch_scene_pairs(c["scenes"])
        ctx.sort_pairs(pairs, count)
        return dict(per_scene=per_scene, count=count, pairs=pairs)
    if kind == "static":
        pairs, count, total = s["pairs"], ctypes.c_int64(), ctypes.c_int64()
        status = s["lib"].stq_sweep_static(s["boxes"].data_ptr(), s["n"], c["axis"], pairs.data_ptr(), pairs.shape[0],
                                           ctypes.byref(count), ctypes.byref(total), s["stream"])
        if status != stq.STQ_OK:
            raise RuntimeError("stq_sweep_static: status %d" % status)
        s["ctx"].sort_pairs(pairs, count.value)
        return dict(count=count.value, pairs=pairs)
    if kind == "host":
        count = _all(s["ctx"].sweep_host(s["boxes"], s["pairs"], axis=c["axis"]))
        s["pairs"][:count].reshape(-1).view(np.int64).sort()
        return dict(count=count, pairs=s["pairs"])
    server = s["server"]
    ids = [server.submit(m, steps, 0.003, seed) for m, steps, seed in s["requests"]]
    done = 0
    while done < len(ids):
        done += len(server.tick())
    results = [server.result(i) for i in ids]
    return dict(counts=np.concatenate([a for a, _ in results]),
                checksums=np.concatenate([b for _, b in results]).view(np.int64))


def exact(case, seed):
    return None  # whole numbers and box bytes only


# ---- what a pass cannot do without --------------------------------------------------

def _grid(g):
    return g * g, 3 * (g - 1) ** 2 + 2 * (g - 1), 2 * (g - 1) ** 2


def _mesh_bytes(boxes):
    """Mesh of a sheet scene with that many boxes (vertices : edges : faces = 1 : 3 : 2):
    two fp64 positions per vertex, index pairs and triples."""
    return boxes * (48 + 3 * 8 + 2 * 12) / 6


def work(case):
    """Inputs read once, outputs written once. Pairs per box are those of the
    scene family (measured on the listed sizes); the count itself is an output."""
    c, kind = case, case["kind"]
    if kind in ("step", "resume", "static"):
        if c["scene"] == "random":
            boxes, pairs = c["boxes"], 0.35e-6 * c["boxes"] ** 2
        else:
            nv, ne, nf = _grid(c["g"])
            boxes = (2 if c["scene"] == "cloth" else c["sheets"]) * (nv + ne + nf)
            pairs = boxes * (4.5 if c["scene"] == "cloth" else 3.2 + 12.3 * max(0, c["g"] - 110) / 140)
        if kind == "static":
            return {"bytes": 44 * boxes + 8 * pairs, "flops": 0}
        return {"bytes": _mesh_bytes(boxes) + 44 * boxes + 8 * pairs, "flops": 0}
    if kind == "batch":
        boxes = c["scenes"] * (c["hi"] - c["lo"]) / math.log(c["hi"] / c["lo"])
        return {"bytes": _mesh_bytes(boxes) + 8 * (4 * boxes + c["scenes"]), "flops": 0}
    if kind == "boxes":
        boxes = c["scenes"] * c["per"]
        return {"bytes": 44 * boxes + 8 * c["scenes"] * (1 + 0.35e-6 * c["per"] ** 2), "flops": 0}
    if kind == "host":
        return {"bytes": 44 * c["boxes"] + 8 * 0.35e-6 * c["boxes"] ** 2, "flops": 0}
    # each step of a request reads its positions and indices, writes the next positions, and gives a count and a checksum
    boxes = c["requests"] * (c["hi"] - c["lo"]) / math.log(c["hi"] / c["lo"]) * (1 + c["max_steps"]) / 2
    return {"bytes": _mesh_bytes(boxes) + 48 * boxes / 6 + 16 * c["requests"] * (1 + c["max_steps"]) / 2, "flops": 0}
