"""A failed or missing job of the bench's serving stream ends the bench: no
latency is made of jobs that were not served."""
import importlib.util
import os

import pytest

from subby_gb300 import serve

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def bench():
    spec = importlib.util.spec_from_file_location("bench", os.path.join(ROOT, "bench.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


def _jobs(n):
    return [serve.Job(id=i, alignment=None, tree=None, model=None) for i in range(n)]


def test_served_jobs_pass(bench):
    jobs = _jobs(3)
    assert bench.all_served(jobs, 3, "stream") is jobs


def test_a_failed_job_ends_the_run(bench):
    jobs = _jobs(3)
    jobs[1].error = "CUDA error (-4)"
    with pytest.raises(RuntimeError, match=r"warm-up: 1 failed jobs, 3 of 3 returned; first: job 1: CUDA error"):
        bench.all_served(jobs, 3, "warm-up")


def test_a_missing_job_ends_the_run(bench):
    with pytest.raises(RuntimeError, match="0 failed jobs, 2 of 3 returned"):
        bench.all_served(_jobs(2), 3, "stream")
