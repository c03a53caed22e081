"""A bounded device wait that gives up is reported by every synchronous call:
gradients, and host-pointer counts, per-branch counts and posteriors.

The hook subby_debug_fail_waits makes the walk's prologue wait on an mbarrier
that nothing arms, with no copy in flight, for a few polls; the walk then
skips its work and returns.  Nothing here faults or hangs the GPU.  With the
hook off the same calls give what they gave before it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import subby_gb300 as sg  # noqa: E402
from subby_gb300 import _lib, synth  # noqa: E402


def _calls(plan, aln):
    return {
        "grad": lambda: plan.grad(aln),
        "run": lambda: list(plan.run(aln, loglike=True, counts=True).values()),
        "branch_counts": lambda: [plan.branch_counts(aln)],
        "posteriors": lambda: list(plan.posteriors(aln, want_branch=True).values()),
        "branch posteriors": lambda: list(plan.posteriors(aln, want_node=False, want_branch=True).values()),
    }


@pytest.mark.parametrize("A,irreversible", [(16, False), (20, False), (32, False), (64, False), (20, True)])
def test_synchronous_calls_report_a_wait_that_gave_up(A, irreversible):
    rng = np.random.default_rng(A)
    model = sg.models.random_irreversible(A, rng) if irreversible else sg.models.random_reversible(A, rng, 0.5, 2.0)[0]
    tree = synth.random_tree(7, 0.1, rng)
    aln = rng.integers(0, A + 2, size=(len(tree.parentIndex), 150)).astype(np.int32)
    plan = sg.Plan(tree, model)
    d_aln = torch.as_tensor(aln).cuda()
    calls = _calls(plan, aln)
    # (node posteriors at A = 16, 20, 32 come from the walk without a ring)
    if A != 64:
        calls["posteriors"]()
        del calls["posteriors"]
    before = {k: [np.array(x) for x in f()] for k, f in calls.items()}
    lib = _lib.load()
    try:
        assert lib.subby_debug_fail_waits(8) == 0
        for k, f in calls.items():
            with pytest.raises(_lib.SubbyError) as e:
                f()
            assert e.value.code == _lib.ERR_TIMEOUT, k
        # device pointers: the status check reports it, once
        plan.run(d_aln, loglike=True, counts=True)
        with pytest.raises(_lib.SubbyError) as e:
            plan.status()
        assert e.value.code == _lib.ERR_TIMEOUT
        plan.status()
    finally:
        lib.subby_debug_fail_waits(0)
    for k, f in calls.items():
        for x, y in zip(f(), before[k]):
            # (the irreversible gradient's FP64 sums have no fixed order)
            tol = 1e-9 if k == "grad" and irreversible else 0
            np.testing.assert_allclose(x, y, rtol=tol, atol=tol * np.abs(y).max())
    plan.status()
    plan.close()
