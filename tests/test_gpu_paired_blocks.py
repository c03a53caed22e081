"""Irreversible counts over conjugate-paired units (k_projx, k_accx) where a CTA
takes several column blocks: more blocks than SMs, with columns of a first, a
later and the short last block against the FP64 oracle, and block sizes that
follow the column count, bit-identical to each other.  The models are
well-conditioned (the route is asserted by the launch count: walk, projection,
accumulation), at A = 32 with eigenvectors that are not orthogonal."""
import numpy as np
import pytest

import oracle
from subby_gb300 import _lib, models, synth
from tests._tol import assert_cols, COUNTS_RTOL

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import subby_gb300 as sg  # noqa: E402


def _cond(m):
    V = np.asarray(m.eigenvectors)
    return np.linalg.cond(V / np.linalg.norm(V, axis=0))


def _model(A, rng):
    """A strong cycle and a few random rates: pairs, eigenvectors close to a
    circulant's but not orthogonal."""
    while True:
        Q = rng.uniform(0.0, 4.0, size=(A, A)) / A
        for a in range(A):
            Q[a, (a + 1) % A] += 2.0
            Q[a, (a + 3) % A] += 0.5
        np.fill_diagonal(Q, 0.0)
        np.fill_diagonal(Q, -Q.sum(axis=1))
        pi = models.stationary_distribution(Q)
        m = models.irrev_model_from_rate_matrix(Q / -np.sum(pi * np.diag(Q)), pi)
        if 1.05 < _cond(m) < 15.0:
            return m


@pytest.mark.parametrize("A", [16, 20, 32])
def test_column_blocks(A):
    rng = np.random.default_rng(A)
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    m = _model(A, rng)
    assert not np.allclose(np.linalg.inv(m.eigenvectors), np.conj(m.eigenvectors).T, atol=1e-3)
    tree = synth.random_tree(6, 0.1, rng)
    most = 2 * 128 * nsm + 37     # (blocks hold at most 128 columns)
    aln = rng.integers(0, A + 2, size=(len(tree.parentIndex), most)).astype(np.int32)
    d = torch.as_tensor(aln).cuda()
    plan = sg.Plan(tree, m)
    full = plan.run(d, loglike=False, counts=True)["counts"]
    assert _lib.last_launch_count() == 3
    # first blocks, second blocks of the first CTAs, the last block
    cols = np.r_[0:6, most // 2:most // 2 + 6, 128 * nsm - 3:128 * nsm + 6, most - 6:most]
    md = dict(eigenvalues=m.eigenvalues, eigenvectors=m.eigenvectors, eigenvectors_inv=m.eigenvectors_inv, pi=m.pi,
              reversible=False)
    ref = oracle.Counts(np.ascontiguousarray(aln[:, cols]), oracle.Tree(tree.parentIndex, tree.distanceToParent), md)
    assert_cols(full.cpu().numpy()[..., cols], ref, COUNTS_RTOL * max(1.0, _cond(m) / 10), "counts")
    # the same columns in blocks of every size
    for C in (1, 17, 16 * nsm, 16 * nsm + 1, 30 * nsm, 50 * nsm + 3):
        part = plan.run(d[:, :C].contiguous(), loglike=False, counts=True)["counts"]
        assert _lib.last_launch_count() == 3
        assert torch.equal(part, full[..., :C]), C
    plan.status()
    plan.close()
