"""The A = 4 inside + outside kernel (k_pass4) against the FP64 oracle: one
branch pair, both program sizes (128 steps and one more), a tree whose tables
leave one CTA per SM, caterpillar and balanced trees (no stack slot, the
deepest stack); one column, a CTA and one more, both sides of the switch to
two columns per thread; every mask and counts kind, and the node posteriors.
Tolerances: the suite's FP32 bars (``_tol``)."""
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


def _tree(kind, leaves, rng):
    if kind == "random":
        return synth.random_tree(leaves, 0.1, rng)
    parent = [-1]
    todo = [(0, leaves)]
    while todo:
        p, k = todo.pop()
        for part in ((1, k - 1) if kind == "caterpillar" else (k // 2, k - k // 2)):
            parent.append(p)
            if part > 1:
                todo.append((len(parent) - 1, part))
    # preorder numbering is not needed: parents come before their children
    return sg.Tree(np.asarray(parent, np.int32), np.concatenate([[0.0], rng.exponential(0.1, len(parent) - 1)]))


def _check(kind, leaves, C, cols, seed, posteriors=True):
    rng = np.random.default_rng(seed)
    t = _tree(kind, leaves, rng)
    pi = rng.dirichlet(np.full(4, 2.0))
    ot = oracle.Tree(t.parentIndex, t.distanceToParent)
    for m, f81 in ((models.hky85_diag(2.0, pi), False), (models.f81_model(pi), True)):
        aln = synth.simulated_alignment(t, m, C, 0.15, rng, unobserved_split=True)
        aln[0, ::5] = rng.integers(0, 4, size=len(aln[0, ::5]))   # observed internal nodes
        md = {"eigenvalues": m.eigenvalues, "eigenvectors": m.eigenvectors, "pi": m.pi}
        sub = aln[:, cols]
        plan = sg.Plan(t, m)
        d = torch.as_tensor(aln).cuda()
        for mask in ("auto", None, rng.random(aln.shape) < 0.7):
            r = plan.run(d, loglike=True, rootprob=True, counts=True, f81=f81, branch_mask=mask)
            om = mask if mask is None or isinstance(mask, str) else mask[:, cols]
            assert_loglike(r["logLike"].cpu().numpy()[cols], oracle.LogLike(sub, ot, md))
            assert_cols(r["rootProb"].cpu().numpy()[:, cols], oracle.RootProb(sub, ot, md), 1e-4, "rootProb")
            assert_cols(r["counts"].cpu().numpy()[:, :, cols],
                        oracle.Counts(sub, ot, md, f81_fast=f81, branch_mask=om), 1e-4, "counts")
        if posteriors:
            got = plan.posteriors(d)["node"].cpu().numpy()[:, :, cols]
            ref = np.asarray(oracle.NodePosterior(sub, ot, md))
            assert np.abs(got - ref).max() <= 1e-4
        plan.close()


@pytest.mark.parametrize("kind,leaves", [("random", 2), ("random", 129), ("random", 130), ("caterpillar", 40),
                                         ("balanced", 64), ("balanced", 512)])
@pytest.mark.parametrize("C", [1, 129])
def test_trees(kind, leaves, C):
    _check(kind, leaves, C, np.arange(C), leaves + C)


@pytest.mark.parametrize("extra", [0, 1, 65])
def test_both_sides_of_two_columns_per_thread(extra):
    C = 384 * torch.cuda.get_device_properties(0).multi_processor_count + extra
    _check("random", 16, C, np.r_[0:70, C // 2:C // 2 + 70, C - 70:C], 7 + extra)


# tables that leave one CTA per SM: whole warps per SM, and a column more
@pytest.mark.parametrize("per_sm", [32, 33, 96])
@pytest.mark.parametrize("extra", [0, 1])
def test_large_tables_in_equal_waves(per_sm, extra):
    C = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + extra
    _check("random", 512, C, np.r_[0:8, C // 2:C // 2 + 8, C - 8:C], per_sm + extra, posteriors=False)
