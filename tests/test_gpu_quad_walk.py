"""The four-lane walk (k_qwalk) and its projection (k_proj): the sizes where
they change form, against the FP64 oracle.

Columns: a lone column, one less / more than a warp's, a CTA's and a
projection tile's, and both sides of the switch from one to two columns per
lane (more columns than 12 warps of 8 per SM).  Trees: one branch pair, a
random one, a caterpillar (a single stored child all the way).  Tolerances
are the suite's FP32 bars (``_tol``): logLike 1e-5, columns 1e-4.
"""
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


def _caterpillar(leaves, rng):
    parent, top = [-1], 0
    for i in range(leaves - 1):   # (leaf, spine) pairs
        parent += [top, top]
        top = len(parent) - 1
    return sg.Tree(np.asarray(parent, np.int32), np.concatenate([[0.0], rng.exponential(0.1, len(parent) - 1)]))


def _case(A, model, tree, C, seed):
    rng = np.random.default_rng(seed)
    t = _caterpillar(7, rng) if tree == "caterpillar" else synth.random_tree({"pair": 2, "random": 9}[tree], 0.2, rng)
    if model == "reversible":
        m = models.random_reversible(A, rng, 0.5, 2.0)[0]
    else:
        m = models.f81_model(rng.dirichlet(np.full(A, 2.0)))
    aln = synth.simulated_alignment(t, m, C, 0.15, rng, unobserved_split=True)
    aln[0, ::5] = rng.integers(0, A, size=len(aln[0, ::5]))   # observed internal nodes
    md = {"eigenvalues": m.eigenvalues, "eigenvectors": m.eigenvectors, "pi": m.pi}
    return aln, t, m, md, oracle.Tree(t.parentIndex, t.distanceToParent)


def _check(aln, t, m, md, ot, cols, f81, mask):
    plan = sg.Plan(t, m)
    d = torch.as_tensor(aln).cuda()
    r = plan.run(d, loglike=True, counts=True, rootprob=True, f81=f81, branch_mask=mask)
    alone = plan.run(d, loglike=True, rootprob=True)   # inside pass only
    torch.cuda.synchronize()
    plan.status()
    sub = aln[:, cols]
    omask = mask if mask is None or isinstance(mask, str) else mask[:, cols]
    ll = oracle.LogLike(sub, ot, md)
    assert_loglike(r["logLike"].cpu().numpy()[cols], ll)
    assert_loglike(alone["logLike"].cpu().numpy()[cols], ll)
    assert_cols(alone["rootProb"].cpu().numpy()[:, cols], oracle.RootProb(sub, ot, md), 1e-4, "rootProb")
    assert_cols(r["counts"].cpu().numpy()[:, :, cols], oracle.Counts(sub, ot, md, f81_fast=f81, branch_mask=omask),
                1e-4, "counts")
    plan.close()


@pytest.mark.parametrize("A", [16, 20, 32])
@pytest.mark.parametrize("tree", ["pair", "random", "caterpillar"])
@pytest.mark.parametrize("C", [1, 7, 33, 129])
def test_few_columns(A, tree, C):
    aln, t, m, md, ot = _case(A, "reversible", tree, C, 10 * A + C)
    rng = np.random.default_rng(C)
    for mask in ("auto", None, rng.random(aln.shape) < 0.7):
        _check(aln, t, m, md, ot, np.arange(C), False, mask)


@pytest.mark.parametrize("A", [16, 20, 32])
@pytest.mark.parametrize("extra", [0, 1, 77])
def test_both_sides_of_two_columns_per_lane(A, extra):
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    C = nsm * 12 * 8 + extra
    aln, t, m, md, ot = _case(A, "reversible", "random", C, A + extra)
    cols = np.r_[0:40, C // 2:C // 2 + 40, C - 40:C]
    _check(aln, t, m, md, ot, cols, False, "auto")


@pytest.mark.parametrize("A", [16, 20, 32, 64])
@pytest.mark.parametrize("C", [1, 45])
def test_closed_form(A, C):
    aln, t, m, md, ot = _case(A, "f81", "random", C, A + C)
    _check(aln, t, m, md, ot, np.arange(C), True, "auto")
    _check(aln, t, m, md, ot, np.arange(C), False, None)


@pytest.mark.parametrize("A", [16, 20, 32])
@pytest.mark.parametrize("C", [1, 37, 4097])
def test_gradient(A, C):
    """Branch-length gradient with weights: fewer branches than a CTA's group
    of them and one left over, column blocks of 4096 and a remainder."""
    for tree in ("pair", "random", "caterpillar"):
        aln, t, m, md, ot = _case(A, "reversible", tree, C, 3 * A + C)
        g = np.random.default_rng(C).integers(1, 5, size=C).astype(np.float64)
        plan = sg.Plan(t, m)
        ll, dt, dS = plan.grad(aln, g)
        plan.close()
        assert_loglike(ll, oracle.LogLike(aln, ot, md))
        ref = oracle.loglike_distance_grad(aln, ot, md, g)
        assert np.abs(dt - ref).max() <= 1e-4 * np.abs(ref).max()
        # V^T dS V = sum_n J_n o X_n and J_n[k][k] = t_n e^{mu_k t_n}, so its
        # mu-weighted trace is sum_n t_n d/dt_n
        V, tn = np.asarray(m.eigenvectors), np.asarray(t.distanceToParent)
        trace = (np.diag(V.T @ dS @ V) * np.asarray(m.eigenvalues)).sum()
        assert abs(trace - (dt * tn).sum()) <= 1e-9 * np.abs(dt * tn).sum()
