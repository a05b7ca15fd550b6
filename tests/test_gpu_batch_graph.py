"""Batches whose runs clear integration buffers first: a job longer than one
launch's 32768 samples is split, its splits add into a cleared buffer, and the
run (clears, then the kernel) is captured and replayed as a graph.  Small jobs
beside it make more items than CTAs, so that the replayed kernel uses the work
queue that each launch leaves zeroed; runs follow one another without a wait."""
import numpy as np
import pytest

from test_gpu_batch import make_jobs

pytestmark = pytest.mark.gpu

SHAPES = [(32, 2, 32768 + 256), (32, 64, 256), (16, 2, 65536 + 16), (64, 96, 128), (96, 11, 384)]


@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("graph", [False, True])
def test_runs_with_clears(xg, oracle_mod, graph, pair):
    import torch
    jobs, keep = make_jobs(torch, oracle_mod, SHAPES, seed0=700)
    exact = [oracle_mod.xengine_i64(x, n, f, t) for x, xd, st, n, f, t in keep]
    torch.cuda.synchronize()
    with xg.Batch(jobs, graph=graph, pair=pair) as b:
        info = b.info()
        assert info["work_items"] > info["grid"]
        for runs in (1, 3):
            for _ in range(runs):
                b.run()
            b.sync()
            for want, (x, xd, st, n, f, t) in zip(exact, keep):
                assert np.array_equal(st.cpu().numpy(), want), (n, f, t)
                st.fill_(7)
            torch.cuda.synchronize()


@pytest.mark.parametrize("pair", [False, True])
def test_clears_keep_accumulating_jobs(xg, oracle_mod, pair):
    """A replayed run clears the buffers of replacing jobs only."""
    import torch
    jobs, keep = make_jobs(torch, oracle_mod, SHAPES, seed0=800)
    for q in (1, 2):
        keep[q][2].zero_()
        jobs[q]["accumulate"] = 1
    torch.cuda.synchronize()
    with xg.Batch(jobs, graph=True, pair=pair) as b:
        for _ in range(3):
            b.run()
        b.sync()
    for q, (x, xd, st, n, f, t) in enumerate(keep):
        want = (3 if q in (1, 2) else 1) * oracle_mod.xengine_i64(x, n, f, t)
        assert np.array_equal(st.cpu().numpy(), want), (n, f, t)
