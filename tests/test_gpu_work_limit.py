"""A = 4 counts and posteriors when the device has no memory for the node
vectors of a full grid: fewer CTAs (the same bits), then the kernel that keeps
them on chip (the oracle's tolerance); an error only when nothing fits, after
which the plan still works."""
import numpy as np
import pytest

import oracle
from tests._tol import assert_cols, assert_loglike, COUNTS_RTOL

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import subby_gb300 as sg  # noqa: E402
from subby_gb300 import _lib, synth  # noqa: E402


def _setup(leaves, C, f81):
    rng = np.random.default_rng(leaves)
    pi = rng.dirichlet(np.full(4, 2.0))
    model = sg.models.f81_model(pi) if f81 else sg.models.hky85_diag(2.0, pi)
    tree = synth.random_tree(leaves, 0.1, rng)
    aln = rng.integers(0, 6, size=(len(tree.parentIndex), C)).astype(np.int32)
    aln[~synth.leaf_mask(tree)] = 4
    return sg.Plan(tree, model), tree, model, aln, torch.as_tensor(aln).cuda()


# (leaves, columns, F81, limit, the same kernel): 128 leaves have 127 steps of
# 20 bytes, so 152 CTAs of 128 threads and two columns take 99 MB (the grid's
# floor for counts); 512 leaves do not fit the on-chip kernel
@pytest.mark.parametrize("leaves,C,f81,limit,same", [
    (128, 120000, False, 110 << 20, True),
    (128, 120000, False, 1 << 20, False),
    (128, 120000, True, 1 << 20, False),
    (512, 20000, False, 20 << 20, True),
])
def test_counts_with_less_memory(leaves, C, f81, limit, same):
    plan, tree, model, aln, d = _setup(leaves, C, f81)
    kw = dict(loglike=True, counts=True, rootprob=True, f81=f81)
    ref = {k: v.cpu() for k, v in plan.run(d, **kw).items()}
    held = plan.device_bytes()
    plan.trim()
    lib = _lib.load()
    try:
        lib.subby_debug_alloc_limit(limit)
        got = {k: v.cpu() for k, v in plan.run(d, **kw).items()}
        assert plan.device_bytes() < held
    finally:
        lib.subby_debug_alloc_limit(0)
    if same:
        assert all(torch.equal(got[k], ref[k]) for k in ref)
    cols = np.r_[0:24, C - 24:C]
    t = oracle.Tree(tree.parentIndex, tree.distanceToParent)
    md = model._asdict()
    assert_loglike(got["logLike"].numpy()[cols], oracle.LogLike(aln[:, cols], t, md))
    assert_cols(got["counts"].numpy()[..., cols], oracle.Counts(aln[:, cols], t, md, f81_fast=f81), COUNTS_RTOL, "counts")
    assert_cols(got["rootProb"].numpy()[..., cols], oracle.RootProb(aln[:, cols], t, md), COUNTS_RTOL, "rootProb")
    plan.close()


def test_posteriors_with_less_memory():
    plan, _, _, _, d = _setup(64, 50000, False)
    ref = {k: v.cpu() for k, v in plan.posteriors(d, want_branch=True).items()}
    plan.trim()
    lib = _lib.load()
    try:
        lib.subby_debug_alloc_limit(8 << 20)
        got = {k: v.cpu() for k, v in plan.posteriors(d, want_branch=True).items()}
        plan.trim()
        lib.subby_debug_alloc_limit(1000)
        with pytest.raises(_lib.SubbyError) as e:
            plan.posteriors(d)
        assert e.value.code == _lib.ERR_NOMEM
    finally:
        lib.subby_debug_alloc_limit(0)
    assert all(torch.equal(got[k], ref[k]) for k in ref)
    again = plan.posteriors(d, want_branch=True)
    assert all(torch.equal(again[k].cpu(), ref[k]) for k in ref)
    plan.close()
