"""Calls of one plan on two streams, enqueued without a host wait between them:
the calls that share the plan's workspace follow one another on the device,
so every result equals its serial call bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import subby_gb300 as sg  # noqa: E402
from subby_gb300 import synth  # noqa: E402


def _counts(plan, aln, stream):
    return plan.run(aln, loglike=True, counts=True, stream=stream)


def _posteriors(plan, aln, stream):
    return plan.posteriors(aln, stream=stream)


def _loglike(plan, aln, stream):
    return plan.run(aln, loglike=True, rootprob=True, stream=stream)


# (alphabet, leaves, columns of the two alignments, the two calls): A = 4 with
# the GPU full and with half of its SMs idle; workspaces that grow between the
# calls; staging walks; a call without workspace beside one with it
CASES = [
    (4, 128, 400000, 400000, _counts, _counts),
    (4, 512, 5000, 4000, _counts, _counts),
    (4, 512, 3000, 5000, _counts, _posteriors),
    (4, 64, 1000, 200000, _counts, _counts),
    (4, 128, 200000, 200000, _counts, _loglike),
    (20, 100, 6000, 7000, _counts, _counts),
    (20, 30, 3000, 3000, _counts, _posteriors),
    (64, 32, 3000, 5000, _counts, _counts),
]


@pytest.mark.parametrize("A,leaves,c0,c1,f0,f1", CASES)
def test_two_streams_of_one_plan(A, leaves, c0, c1, f0, f1):
    rng = np.random.default_rng([A, leaves])
    model = sg.models.hky85_diag(2.0, [0.1, 0.2, 0.3, 0.4]) if A == 4 else sg.models.random_reversible(A, rng, 0.5, 2.0)[0]
    tree = synth.random_tree(leaves, 0.1, rng)
    R = len(tree.parentIndex)
    alns = []
    for C in (c0, c1):
        a = torch.as_tensor(rng.integers(0, A + 2, size=(R, C)).astype(np.int32)).cuda()
        a[~torch.as_tensor(synth.leaf_mask(tree))] = A
        alns.append(a)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    calls = [(f0, alns[0]), (f1, alns[1])]
    ref = []
    for f, a in calls:
        plan = sg.Plan(tree, model)
        torch.cuda.synchronize()
        r = f(plan, a, streams[0])
        torch.cuda.synchronize()
        ref.append({k: v.cpu() for k, v in r.items()})
        plan.close()
    plan = sg.Plan(tree, model)
    h_aln = alns[0][:, :500].cpu().numpy()
    h_ref = plan.run(h_aln, loglike=True, counts=True)
    plan.trim()
    for _ in range(3):
        got = [f(plan, a, streams[i % 2]) for i, (f, a) in enumerate(calls * 2)]
        # (host pointers on the default stream, behind both)
        host = plan.run(h_aln, loglike=True, counts=True)
        torch.cuda.synchronize()
        for i, r in enumerate(got):
            for k in ref[i % 2]:
                assert torch.equal(r[k].cpu(), ref[i % 2][k]), (i, k)
        for k in h_ref:
            assert np.array_equal(host[k], h_ref[k]), k
        plan.trim()
    plan.close()
