"""Handles of different sizes in different threads at the same time: each builds its run graph (the kernels' shared
memory limit is common to them) and runs the cooperative kernels beside the other's."""

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def system(n, seed=1):
    import frictionqpotspringblock_gb300 as fqsb

    s = fqsb.Line1d.System_Cuspy_Laplace(m=1.0, eta=0.1, mu=1.0, k_interactions=1.0, k_frame=1.0 / n, dt=0.1, shape=[n],
                                         seed=seed, distribution="weibull", parameters=[2.0, 1.0, 1e-5], offset=-5.0,
                                         nchunk=34)
    s.u = np.random.default_rng(n).normal(0.0, 0.2, n)
    return s


def grid(rows, cols):
    import frictionqpotspringblock_gb300 as fqsb

    s = fqsb.Line2d.System_Cuspy_Laplace(m=1.0, eta=0.2, mu=1.0, k_interactions=1.0, k_frame=0.01, dt=0.1,
                                         shape=[rows, cols], seed=5, distribution="weibull", parameters=[2.0, 1.0, 1e-5],
                                         offset=-5.0, nchunk=34)
    s.u = np.random.default_rng(rows).normal(0.0, 0.2, (rows, cols))
    return s


def ensemble():
    from frictionqpotspringblock_gb300 import batch

    n = np.array([300, 2000, 77, 5000])
    b = batch.Line1d_System_Cuspy_Laplace(n, 7 + np.arange(4), 1.0 / n, m=1.0, eta=0.1, mu=1.0, k_interactions=1.0, dt=0.1,
                                          distribution="weibull", parameters=[2.0, 1.0, 1e-5], offset=-5.0, nchunk=100,
                                          window=64)
    b.quasistatic(1, 1e-5)
    return np.concatenate([b.field(j) for j in range(4)])


def strips():
    """Sizes of the shortest and the longest strips."""
    out = []
    for n in (5000, 2 ** 21 + 3, 40000, 600000):
        s = system(n)
        s.flowSteps(30, 0.5)
        s.minimise(max_iter=20, max_iter_is_error=False)
        out.append(s.u)
    return out


def long_run():
    s = system(2 ** 20)
    s.flowSteps(3000, 0.5)
    return [s.u]


def grids():
    out = []
    for shape in ((70, 61), (400, 300)):
        s = grid(*shape)
        s.flowSteps(300, 0.5)
        s.minimise(max_iter=300, max_iter_is_error=False)
        out.append(s.u)
    return out


@pytest.mark.parametrize("jobs", [(strips, strips), (strips, long_run), (grids, long_run), (ensemble, long_run),
                                  (ensemble, grids, strips)])
def test_at_the_same_time(jobs):
    alone = [job() for job in jobs]
    got, errors = [None] * len(jobs), []
    start = threading.Barrier(len(jobs))

    def work(k):
        try:
            start.wait()
            got[k] = [jobs[k]() for _ in range(3)]
        except Exception as e:  # noqa: BLE001 -- reported below, in the test's own thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for a, bs in zip(alone, got):
        for b in bs:
            for x, y in zip(a, b):
                assert np.array_equal(x, y)
