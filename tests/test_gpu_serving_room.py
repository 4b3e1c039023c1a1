"""FP64 serving under a budget that holds the structures but not the tensor-core
kernels' tables: every structure is admitted as if those tables did not exist, the
budget is kept, and results are the job's own."""
import numpy as np
import pytest

import lcpgrid as L

pytestmark = pytest.mark.gpu


def _results(srv, n):
    out = {}
    while len(out) < n:
        for tag, e, _ in srv.poll(wait_ms=2000):
            out[tag] = e
    return out


@pytest.mark.parametrize("room", [1.02, 2.5, 30.0])
def test_tables_keep_no_structure_out(room):
    from test_gpu_serving import _structures
    ctx = L.Context(0)
    jobs = _structures(ctx)
    base = [job.footprint() for job, _ in jobs]
    budget = int(room * sum(base))
    srv = L.Server(0, nslots=2, precision="fp64", budget_bytes=budget)
    ids = [srv.add(job) for job, _ in jobs]
    assert [srv.state(i) for i in ids] == [L.Server.ADMITTED] * len(ids)
    for _ in range(2):
        for i, (_, dm) in zip(ids, jobs):
            srv.submit(i, dm, tag=i)
        got = _results(srv, len(ids))
    assert srv.stats()[2] <= budget
    held = [job.footprint() for job, _ in jobs]
    assert (sum(held) > sum(base)) == (room > 1.5)  # the tables are made where they fit
    srv.close()
    for i, (job, dm) in zip(ids, jobs):
        job.set_dm(dm)
        job.step()
        np.testing.assert_allclose(got[i], job.energies(), rtol=1e-12)
