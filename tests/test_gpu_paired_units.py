"""Irreversible counts over conjugate-paired units (k_projx, k_accx) at A =
16, 20, 32 against the FP64 oracle: eigensystems with pairs and reals, with
reals only (a reversible matrix in irreversible form), pairs with orthogonal
eigenvectors (a circulant matrix; the random ones are often too ill-conditioned
at A = 32 for the units) and one that is not in conjugate form (its columns
carry phases: the general kernel); one column, a
block of columns and one more, more branches than one run of the register
sums.  Tolerance: the irreversible bar, 1e-4 x max(1, cond(V) / 10)."""
import numpy as np
import pytest

import oracle
from subby_gb300 import models, synth
from subby_gb300.types import IrrevDiagModel
from tests._tol import assert_cols

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import subby_gb300 as sg  # noqa: E402


def _model(A, kind, rng):
    if kind == "reals":
        _, log_exch, pi = models.random_reversible(A, rng, 0.5, 2.0)
        return models.irrev_model_from_rate_matrix(models.reversible_rate_matrix(log_exch, pi), pi)
    if kind == "circulant":
        r = rng.gamma(1.0, size=A)
        r[0] = 0.0
        Q = np.stack([np.roll(r, i) for i in range(A)]) / r.sum()
        np.fill_diagonal(Q, -1.0)
        return models.irrev_model_from_rate_matrix(Q, np.full(A, 1.0 / A))
    m = models.random_irreversible(A, rng)
    if kind == "phases":
        f = np.exp(1j * rng.uniform(0, 2 * np.pi, A)) * rng.uniform(0.5, 2.0, A)
        m = IrrevDiagModel(m.eigenvalues, m.eigenvectors * f[None, :], m.eigenvectors_inv / f[:, None], m.pi)
    return m


@pytest.mark.parametrize("A", [16, 20, 32])
@pytest.mark.parametrize("kind", ["pairs", "reals", "circulant", "phases"])
@pytest.mark.parametrize("leaves,C", [(2, 1), (9, 129), (40, 57)])
def test_counts(A, kind, leaves, C):
    rng = np.random.default_rng(A + leaves)
    m = _model(A, kind, rng)
    t = synth.random_tree(leaves, 0.1, rng)
    aln = synth.simulated_alignment(t, m, C, 0.1, rng, unobserved_split=True)
    md = dict(eigenvalues=m.eigenvalues, eigenvectors=m.eigenvectors, eigenvectors_inv=m.eigenvectors_inv, pi=m.pi,
              reversible=False)
    ot = oracle.Tree(t.parentIndex, t.distanceToParent)
    tol = 1e-4 * max(1.0, np.linalg.cond(m.eigenvectors) / 10)
    plan = sg.Plan(t, m)
    d = torch.as_tensor(aln).cuda()
    for exact in (False, True):
        for mask in ("auto", None, rng.random(aln.shape) < 0.7):
            r = plan.run(d, loglike=False, counts=True, branch_mask=mask, exact_irreversible=exact)["counts"]
            assert_cols(r.cpu().numpy(), oracle.Counts(aln, ot, md, branch_mask=mask, irrev_exact=exact), tol, "counts")
    plan.status()
    plan.close()
