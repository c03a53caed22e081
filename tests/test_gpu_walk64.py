"""The A = 64 tensor-core walk's coalesced rows and deferred leaf products
against the FP64 oracle: a lone column, one less / more than a warp's and a
tile's columns, two tiles; a root with two leaves (its products are read after
the last step), one leaf per step (caterpillar), none or two (balanced), and a
random tree; every mask.  Tolerances: the suite's FP32 bars (``_tol``)."""
import numpy as np
import pytest

import oracle
from subby_gb300 import models, synth
from tests._tol import assert_cols, assert_loglike

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import subby_gb300 as sg  # noqa: E402


def _tree(kind, rng):
    if kind == "random":
        return synth.random_tree(9, 0.2, rng)
    parent, todo = [-1], [(0, {"pair": 2, "caterpillar": 7, "balanced": 8}[kind])]
    while todo:
        p, k = todo.pop()
        for part in ((1, k - 1) if kind == "caterpillar" else (k // 2, k - k // 2)):
            parent.append(p)
            if part > 1:
                todo.append((len(parent) - 1, part))
    return sg.Tree(np.asarray(parent, np.int32), np.concatenate([[0.0], rng.exponential(0.1, len(parent) - 1)]))


@pytest.mark.parametrize("kind", ["pair", "caterpillar", "balanced", "random"])
@pytest.mark.parametrize("C", [1, 31, 33, 127, 129])
def test_rows_and_leaves(kind, C):
    rng = np.random.default_rng(64 + C)
    t = _tree(kind, rng)
    m = models.random_reversible(64, rng, 0.5, 2.0)[0]
    aln = synth.simulated_alignment(t, m, C, 0.15, rng, unobserved_split=True)
    aln[0, ::5] = rng.integers(0, 64, size=len(aln[0, ::5]))   # observed internal nodes
    md = {"eigenvalues": m.eigenvalues, "eigenvectors": m.eigenvectors, "pi": m.pi}
    ot = oracle.Tree(t.parentIndex, t.distanceToParent)
    plan = sg.Plan(t, m)
    d = torch.as_tensor(aln).cuda()
    for mask in ("auto", None, rng.random(aln.shape) < 0.7):
        r = plan.run(d, loglike=True, rootprob=True, counts=True, branch_mask=mask)
        torch.cuda.synchronize()
        plan.status()
        assert_loglike(r["logLike"].cpu().numpy(), oracle.LogLike(aln, ot, md))
        assert_cols(r["rootProb"].cpu().numpy(), oracle.RootProb(aln, ot, md), 1e-4, "rootProb")
        assert_cols(r["counts"].cpu().numpy(), oracle.Counts(aln, ot, md, branch_mask=mask), 1e-4, "counts")
    plan.close()
