"""Footprint estimates of irreversible serving jobs cover the staging of the
paired-unit counts: raw and projected vectors, the latter in padded blocks."""
import numpy as np
import pytest

from subby_gb300 import models, serve, synth


@pytest.mark.parametrize("A", [16, 20, 32])
def test_irreversible_staging_is_counted(A):
    R, C = 99, 4000
    got = serve.job_device_bytes(R, C, A, irreversible=True)
    raw = serve.job_device_bytes(R, C, A)
    for pairs in range(A // 2 + 1):
        units = (A - pairs + 1) // 2 * 2
        for block in range(8, 129, 8):
            blocks = -(-C // block)
            projected = 8 * (R - 1) * blocks * 2 * units * (block + 2)
            assert got >= raw + projected, (pairs, block)
    # capped per plan like the raw staging
    assert serve.job_device_bytes(R, 1 << 22, A, irreversible=True) == serve.job_device_bytes(R, 1 << 22, A)


def test_jobs_are_admitted_by_their_model():
    rng = np.random.default_rng(3)
    tree = synth.random_tree(30, 0.1, rng)
    aln = np.zeros((59, 700), np.int32)
    need = {}
    for name, m in (("rev", models.random_reversible(20, rng)[0]), ("irr", models.random_irreversible(20, rng))):
        need[name] = serve.Server._bytes(serve.Job(id=0, alignment=aln, tree=tree, model=m))
    assert need["rev"] == serve.job_device_bytes(59, 700, 20)
    assert need["irr"] == serve.job_device_bytes(59, 700, 20, True) > need["rev"]
