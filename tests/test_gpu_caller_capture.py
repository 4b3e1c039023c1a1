"""A caller's own CUDA graph of an FP64 step: it stays valid when a larger cell on the
same context needs larger workspaces, which the step's kernels share."""
import numpy as np
import pytest

import lcpgrid as L

pytestmark = pytest.mark.gpu


def test_captured_step_outlives_workspace_growth():
    torch = pytest.importorskip("torch")
    from test_gpu_parity import psd_dm
    from test_gpu_tc import _mixed_cell, _si2
    ctx = L.Context(0)
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    ctx.set_step_graphs(False)
    u, orbs = _mixed_cell(ctx)
    dm, dm2 = psd_dm(u, 51), psd_dm(u, 52)
    job = L.GridStepJob(u, orbs, "off", "LDA")
    want = []
    for d in (dm, dm2):
        job.set_dm(d)
        job.step()
        want.append((job.hks()[0], job.density()[0]))
    ctx.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        job.step()
    u2, orbs2 = _si2(ctx)
    big = L.GridStepJob(u2, orbs2, "off", "LDA")
    assert u2.Total_Hsize > 2 * u.Total_Hsize
    dm_big = psd_dm(u2, 53)
    big.set_dm(dm_big)
    big.step()
    h_big = big.hks()[0]
    for k, d in enumerate((dm, dm2)):
        job.set_dm(d)
        ctx.synchronize()
        with torch.cuda.stream(stream):
            graph.replay()
        for got, ref in zip((job.hks()[0], job.density()[0]), want[k]):
            np.testing.assert_allclose(got, ref, rtol=1e-12, atol=1e-14 * np.max(np.abs(ref)))
    big.step()  # and the larger cell's workspaces are its own
    np.testing.assert_allclose(big.hks()[0], h_big, rtol=1e-12, atol=1e-14 * np.max(np.abs(h_big)))
