"""The A = 4 inside-only kernel (k_inside4) against the FP64 oracle: one node,
one branch pair, a caterpillar (no stack slot), a balanced tree (the deepest
stack) and a random one; one column, a CTA and one more, both sides of the
switch to two columns per thread; observed internal nodes; and the same
likelihoods as the Counts kernel's inside pass, bit for bit.  Tolerances: the
suite's FP32 bars (``_tol``)."""
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
    if kind == "node":
        return sg.Tree(np.array([-1], np.int32), np.zeros(1))
    if kind == "random":
        return synth.random_tree(33, 0.1, rng)
    parent = [-1]

    def split(p, leaves):
        for k in ((1, leaves - 1) if kind == "caterpillar" else (leaves // 2, leaves - leaves // 2)):
            parent.append(p)
            me = len(parent) - 1
            if k > 1:
                split(me, k)
    split(0, {"pair": 2, "caterpillar": 20, "balanced": 64}[kind])
    return sg.Tree(np.asarray(parent, np.int32), np.concatenate([[0.0], rng.exponential(0.1, len(parent) - 1)]))


def _check(kind, C, cols, seed):
    rng = np.random.default_rng(seed)
    t = _tree(kind, rng)
    m = models.hky85_diag(2.0, rng.dirichlet(np.full(4, 2.0)))
    aln = rng.integers(0, 6, size=(len(t.parentIndex), C)).astype(np.int32)   # every code, internal nodes too
    if kind != "node":
        aln[np.asarray(t.parentIndex[1:])] = np.where(rng.random((len(t.parentIndex) - 1, C)) < 0.1,
                                                      aln[np.asarray(t.parentIndex[1:])], 4)
    md = {"eigenvalues": m.eigenvalues, "eigenvectors": m.eigenvectors, "pi": m.pi}
    ot = oracle.Tree(t.parentIndex, t.distanceToParent)
    plan = sg.Plan(t, m)
    d = torch.as_tensor(aln).cuda()
    r = plan.run(d, loglike=True, rootprob=True)
    full = plan.run(d, loglike=True, rootprob=True, counts=True)
    assert torch.equal(r["logLike"], full["logLike"]) and torch.equal(r["rootProb"], full["rootProb"])
    assert_loglike(r["logLike"].cpu().numpy()[cols], oracle.LogLike(aln[:, cols], ot, md))
    assert_cols(r["rootProb"].cpu().numpy()[:, cols], oracle.RootProb(aln[:, cols], ot, md), 1e-4, "rootProb")
    plan.close()


@pytest.mark.parametrize("kind", ["node", "pair", "caterpillar", "balanced", "random"])
@pytest.mark.parametrize("C", [1, 31, 65, 257])
def test_small(kind, C):
    _check(kind, C, np.arange(C), C)


@pytest.mark.parametrize("extra", [0, 1, 33])
def test_both_sides_of_two_columns_per_thread(extra):
    C = 1024 * torch.cuda.get_device_properties(0).multi_processor_count + extra
    _check("balanced", C, np.r_[0:70, C // 2:C // 2 + 70, C - 70:C], 5 + extra)
