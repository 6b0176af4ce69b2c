"""The sort's waits between blocks, in a build of the library whose blocks give up at
once: the call returns STQ_ERR_TIMEOUT, the kernels after the sort do nothing (the
output stays as it was), and the context goes on working."""
import ctypes
import importlib
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture()
def impatient(pkg, stq, cuda, tmp_path, monkeypatch):
    build = importlib.import_module(pkg.__name__ + ".build")
    obj, lib = tmp_path / "radix_sort.o", tmp_path / "libstq_impatient.so"
    subprocess.run([build._nvcc(), *build.NVCC_FLAGS, "-DSTQ_SORT_POLL_LIMIT=0", "-c", str(build.CSRC / "radix_sort.cu"),
                    "-o", str(obj)], check=True, capture_output=True)
    others = [build.OUT / (s.rsplit(".", 1)[0] + ".o") for s in build.CUDA_SOURCES if s != "radix_sort.cu"]
    subprocess.run([build._nvcc(), build.GENCODE, "-shared", "-Xcompiler", "-fPIC", str(obj), *map(str, others), "-o",
                    str(lib)], check=True, capture_output=True)
    monkeypatch.setattr(stq, "LIB_PATH", lib)
    monkeypatch.setattr(stq, "_lib", None)
    import torch

    with stq.Context(0, torch.cuda.current_stream(cuda).cuda_stream) as c:
        yield c


def dev(a, cuda):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a)).to(cuda)


def test_a_wait_that_runs_out_is_an_error_and_nothing_else(impatient, stq, oracle, cuda):
    import torch

    ctx, n = impatient, 120_000
    boxes = stq.random_boxes(n, seed=11)
    d = dev(boxes.view(np.int32).reshape(-1, 11), cuda)
    few = stq.random_boxes(300, sliver_frac=0.0, seed=12)
    c = 0.5 * (few["min"] + few["max"])
    few["min"], few["max"] = c - np.float32(0.1), c + np.float32(0.1)
    dfew, want = dev(few.view(np.int32).reshape(-1, 11), cuda), oracle.broadphase(few)
    assert len(want) > 100
    pairs = torch.full((1 << 20, 2), -7, dtype=torch.int32, device=cuda)
    m = stq.cloth_pair(g=60, z_offset=0.01, sigma=0.004, seed=21)
    mesh = [dev(x, cuda) for x in (m.V0, m.V1, m.E, m.F)]
    off = [np.array([0, len(x)], np.int64) for x in (m.V0, m.E, m.F)]
    for call in (
        lambda: ctx.sweep(d, n, pairs, 1 << 20),  # the first: prepare, then sweep
        lambda: ctx.sweep(d, n, pairs, 1 << 20),  # queued whole
        lambda: (ctx.prepare(d, n), ctx.sweep_prepared(pairs, 1 << 20)),
        lambda: ctx.batch_broadphase(mesh[0], mesh[1], off[0], mesh[2], off[1], mesh[3], off[2], pairs, 1 << 20),
    ):
        with pytest.raises(stq.STQError) as e:
            call()
        assert e.value.status == stq.STQ_ERR_TIMEOUT
        assert bool((pairs == -7).all())
        got = torch.empty((len(want) + 16, 2), dtype=torch.int32, device=cuda)
        r = ctx.sweep(dfew, len(few), got, len(want) + 16)  # one tile: no wait
        assert np.array_equal(oracle.canonical(got[: r.count].cpu().numpy()), want)


def test_a_wait_that_runs_out_in_the_static_sweep(impatient, stq, cuda):
    import torch

    n = 60_000
    d = dev(stq.random_boxes(n, seed=13).view(np.int32).reshape(-1, 11), cuda)
    pairs = torch.full((1 << 20, 2), -7, dtype=torch.int32, device=cuda)
    count, total = ctypes.c_int64(), ctypes.c_int64()
    st = stq.load_library().stq_sweep_static(d.data_ptr(), n, 0, pairs.data_ptr(), 1 << 20, ctypes.byref(count),
                                             ctypes.byref(total), torch.cuda.current_stream(cuda).cuda_stream)
    assert st == stq.STQ_ERR_TIMEOUT and bool((pairs == -7).all())


def test_a_wait_that_runs_out_in_a_pair_sort(impatient, stq, cuda):
    import torch

    n = 50_000  # of one first id: sorted by digits
    pairs = torch.zeros((n, 2), dtype=torch.int32, device=cuda)
    pairs[:, 1] = torch.arange(n, device=cuda).flip(0)
    with pytest.raises(stq.STQError) as e:
        impatient.sort_pairs(pairs, n)
    assert e.value.status == stq.STQ_ERR_TIMEOUT
    few = pairs[:1000].clone()
    impatient.sort_pairs(few, 1000)
    assert torch.equal(few[:, 1], torch.sort(few[:, 1])[0])
