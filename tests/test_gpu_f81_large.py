"""F81 counts at large alphabets beyond one wave.

A = 64: CTAs of k_acc_f81 that take a second and a short last group of eight
columns, over more branches than two blocks of its scalar buffers (64 each).
A = 16, 20, 32: the closed-form walk with two columns per lane (more than 96
columns per SM).  Sampled columns against the FP64 oracle, at the suite's FP32
tolerances."""
import numpy as np
import pytest

import oracle
from subby_gb300 import models, synth
from tests._tol import assert_cols, assert_loglike, COUNTS_RTOL

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import subby_gb300 as sg  # noqa: E402


def _setup(A, leaves, C):
    rng = np.random.default_rng([A, C])
    model = models.f81_model(rng.dirichlet(np.full(A, 2.0)))
    tree = synth.random_tree(leaves, 0.1, rng)
    aln = rng.integers(0, A + 2, size=(len(tree.parentIndex), C)).astype(np.int32)
    aln[(~synth.leaf_mask(tree))[:, None] & (rng.random(aln.shape) < 0.95)] = A   # a few observed internal nodes
    return rng, model, tree, aln


def _check(plan, model, tree, aln, cols, mask):
    r = plan.run(torch.as_tensor(aln).cuda(), loglike=True, rootprob=True, counts=True, f81=True, branch_mask=mask)
    plan.status()
    sub = np.ascontiguousarray(aln[:, cols])
    t, md = oracle.Tree(tree.parentIndex, tree.distanceToParent), model._asdict()
    om = mask if mask is None or isinstance(mask, str) else mask[:, cols]
    assert_loglike(r["logLike"].cpu().numpy()[cols], oracle.LogLike(sub, t, md))
    assert_cols(r["counts"].cpu().numpy()[..., cols], oracle.Counts(sub, t, md, f81_fast=True, branch_mask=om),
                COUNTS_RTOL, "counts")


@pytest.mark.parametrize("leaves", [33, 70])   # 64 and 138 branches
def test_second_groups_at_64(leaves):
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    C = 16 * nsm + 5
    rng, model, tree, aln = _setup(64, leaves, C)
    cols = np.r_[0:3, 8 * nsm - 2:8 * nsm + 10, C - 7:C]
    plan = sg.Plan(tree, model)
    for mask in ("auto", None, rng.random(aln.shape) < 0.7):
        _check(plan, model, tree, aln, cols, mask)
    plan.close()


@pytest.mark.parametrize("A", [16, 20, 32])
@pytest.mark.parametrize("leaves", [2, 21])
def test_two_columns_per_lane(A, leaves):
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    C = 96 * nsm + 1
    rng, model, tree, aln = _setup(A, leaves, C)
    cols = np.r_[0:18, 64 * nsm - 9:64 * nsm + 9, C - 9:C]
    plan = sg.Plan(tree, model)
    for mask in ("auto", rng.random(aln.shape) < 0.7):
        _check(plan, model, tree, aln, cols, mask)
    # inside only
    r = plan.run(torch.as_tensor(aln).cuda(), loglike=True, rootprob=True)
    sub = np.ascontiguousarray(aln[:, cols])
    t, md = oracle.Tree(tree.parentIndex, tree.distanceToParent), model._asdict()
    assert_loglike(r["logLike"].cpu().numpy()[cols], oracle.LogLike(sub, t, md))
    assert_cols(r["rootProb"].cpu().numpy()[:, cols], oracle.RootProb(sub, t, md), COUNTS_RTOL, "rootProb")
    plan.close()
