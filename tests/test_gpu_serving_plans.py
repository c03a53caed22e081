"""More packed jobs at once than the serving engine caches plans: every plan of
a batch stays until its launch is over, so each result equals its single call
bit for bit, and the cache is back at its limit once the engine is idle."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import subby_gb300 as sg  # noqa: E402
from subby_gb300 import synth, serve  # noqa: E402


@pytest.mark.parametrize("cap", [1, 8])
def test_batches_larger_than_the_plan_cache(cap):
    rng = np.random.default_rng(31)
    jobs = []
    for i in range(48):
        if i < 40:
            tree = synth.random_tree(int(rng.integers(3, 40)), 0.1, rng)
            model = sg.models.hky85_diag(2.0, rng.dirichlet(np.ones(4)))
        else:   # further columns of earlier jobs' trees
            tree, model = jobs[i - 40].tree, jobs[i - 40].model
        aln = synth.simulated_alignment(tree, model, int(rng.integers(1, 1500)), 0.1, rng)
        pin = torch.empty(aln.shape, dtype=torch.int32, pin_memory=True)
        pin.numpy()[:] = aln
        j = serve.Job(id=i, alignment=pin, tree=tree, model=model, f81=(i % 8 == 5),
                      want=("logLike",) if i % 8 == 6 else ("logLike", "counts"))
        j.host = aln
        jobs.append(j)
    srv = serve.NativeServer(max_inflight=4, device_budget=1 << 30, plan_cache=cap)
    done = srv.run(jobs, realtime=False)
    assert len(done) == len(jobs) and srv.stats()["packed_jobs"] == len(jobs)
    for j in done:
        assert not j.error, f"job {j.id}: {j.error}"
        plan = sg.Plan(j.tree, j.model)
        ref = plan.run(j.host, loglike=True, counts="counts" in j.want, f81=j.f81)
        plan.close()
        for k in j.want:
            np.testing.assert_array_equal(j.result[k], ref[k])
        j.release()
    for _ in range(1000):   # the engine publishes its counters once per turn
        if srv.stats()["plans_cached"] <= cap:
            break
        time.sleep(0.01)
    assert srv.stats()["plans_cached"] <= cap
    srv.close()
