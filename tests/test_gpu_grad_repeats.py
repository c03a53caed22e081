"""Gradients of up to 4096 columns are the same in every call, bit for bit:
every FP64 sum has a fixed order.  (More columns: a sum of blocks of 4096 in
no fixed order.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import subby_gb300 as sg  # noqa: E402
from subby_gb300 import synth  # noqa: E402


@pytest.mark.parametrize("A,leaves,C", [(16, 100, 4096), (16, 3, 33), (20, 100, 4096), (20, 2, 1), (32, 60, 4096),
                                        (32, 5, 700), (64, 20, 600)])
def test_repeated_gradients_are_identical(A, leaves, C):
    rng = np.random.default_rng([A, C])
    model = sg.models.random_reversible(A, rng, 0.5, 2.0)[0]
    tree = synth.random_tree(leaves, 0.1, rng)
    aln = synth.simulated_alignment(tree, model, C, 0.1, rng)
    g = rng.integers(1, 5, size=C).astype(np.float32)
    plan = sg.Plan(tree, model)
    first = plan.grad(aln, g)
    for _ in range(8):
        for x, y in zip(plan.grad(aln, g), first):
            np.testing.assert_array_equal(x, y)
    plan.close()
