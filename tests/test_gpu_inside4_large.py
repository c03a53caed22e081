"""LogLike / RootProb of A = 4 trees whose tables leave one CTA per SM: column
counts on both sides of a wave of 32, 160 and 256 threads per SM, bit-identical
to short calls and, on a few columns, within the oracle's tolerance."""
import numpy as np
import pytest

import oracle
from tests._tol import assert_cols, assert_loglike, ROOTPROB_RTOL

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import subby_gb300 as sg  # noqa: E402
from subby_gb300 import synth  # noqa: E402


@pytest.mark.parametrize("leaves", [640, 1100])
def test_large_tables_equal_short_calls(leaves):
    rng = np.random.default_rng(leaves)
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    model = sg.models.hky85_diag(2.0, rng.dirichlet(np.full(4, 2.0)))
    tree = synth.random_tree(leaves, 0.1, rng)
    most = 512 * nsm + 7
    aln = rng.integers(0, 6, size=(len(tree.parentIndex), most)).astype(np.int32)
    aln[~synth.leaf_mask(tree)] = 4
    d = torch.as_tensor(aln).cuda()
    plan = sg.Plan(tree, model)
    t = oracle.Tree(tree.parentIndex, tree.distanceToParent)
    for C in (1, 32 * nsm, 32 * nsm + 1, 160 * nsm - 3, 160 * nsm + 1, 256 * nsm + 1, most):
        r = plan.run(d[:, :C].contiguous(), loglike=True, rootprob=True)
        for c0 in sorted({0, C // 2, max(C - 70, 0)}):
            cols = slice(c0, min(c0 + 70, C))
            s = plan.run(d[:, cols].contiguous(), loglike=True, rootprob=True)
            assert torch.equal(r["logLike"][cols], s["logLike"]) and torch.equal(r["rootProb"][:, cols], s["rootProb"])
    cols = np.r_[0:8, most - 8:most]
    assert_loglike(r["logLike"].cpu().numpy()[cols], oracle.LogLike(aln[:, cols], t, model._asdict()))
    assert_cols(r["rootProb"].cpu().numpy()[:, cols], oracle.RootProb(aln[:, cols], t, model._asdict()), ROOTPROB_RTOL,
                "rootProb")
    plan.close()
