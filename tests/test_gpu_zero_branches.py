"""F81 / JC models on trees with zero-length branches, and columns in which the
two leaves of a zero-length cherry contradict one another.  The closed-form
walk keeps such a column finite, as the eigensystem's tables can: its counts
are those of some history (the dwell times add up to the tree's length,
unmasked); the other columns are the oracle's at the suite's tolerances."""
import numpy as np
import pytest

import oracle
from subby_gb300 import models, synth
from subby_gb300.types import Tree
from tests._tol import assert_cols, assert_loglike, COUNTS_RTOL

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import subby_gb300 as sg  # noqa: E402


@pytest.mark.parametrize("A", [16, 20, 32, 64])
@pytest.mark.parametrize("leaves", [2, 12, 40])
@pytest.mark.parametrize("jc", [False, True])
def test_contradicting_cherry(A, leaves, jc):
    rng = np.random.default_rng([A, leaves, jc])
    model = models.jukes_cantor_model(A) if jc else models.f81_model(rng.dirichlet(np.full(A, 3.0)))
    t = synth.random_tree(leaves, 0.1, rng)
    R = len(t.parentIndex)
    leaf = synth.leaf_mask(t)
    # one cherry and the branches of some internal nodes have length 0
    dist = t.distanceToParent.copy()
    dist[~leaf & (rng.random(R) < 0.4)] = 0.0
    a = next(n for n in range(1, R - 1) if leaf[n] and leaf[n + 1] and t.parentIndex[n] == t.parentIndex[n + 1])
    dist[a:a + 2] = 0.0
    tree = Tree(t.parentIndex, dist)
    C = 150
    aln = np.full((R, C), A, np.int32)
    aln[leaf] = rng.integers(0, A, size=(int(leaf.sum()), C))
    aln[a + 1, ::3] = aln[a, ::3]
    same = aln[a] == aln[a + 1]
    assert same.any() and not same.all()
    d = torch.as_tensor(aln).cuda()
    plan = sg.Plan(tree, model)
    ot, md = oracle.Tree(tree.parentIndex, tree.distanceToParent), model._asdict()
    sub = np.ascontiguousarray(aln[:, same])
    for f81 in (True, False):
        if A == 64 and not f81:
            continue   # (the general tables)
        r = plan.run(d, loglike=True, rootprob=True, counts=True, f81=f81, branch_mask=None)
        ll, rp, ct = (r[k].cpu().numpy() for k in ("logLike", "rootProb", "counts"))
        assert np.isfinite(ll).all() and np.isfinite(rp).all() and np.isfinite(ct).all()
        np.testing.assert_allclose(rp.sum(0), 1.0, atol=1e-4)
        dwell = np.einsum("iic->c", ct.astype(np.float64))
        np.testing.assert_allclose(dwell, dist.sum(), rtol=1e-3, atol=1e-5)
        assert_loglike(ll[same], oracle.LogLike(sub, ot, md))
        assert_cols(ct[..., same], oracle.Counts(sub, ot, md, f81_fast=f81, branch_mask=None), COUNTS_RTOL, "counts")
    ll = plan.run(d, loglike=True)["logLike"].cpu().numpy()
    assert np.isfinite(ll).all()
    plan.close()
