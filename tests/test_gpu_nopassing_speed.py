"""The no-passing minimiser's launch shape (csrc/fqsb_step.cu, build_nopass_graph): a sweep of 2^17 particles against
one of 2^20, which do not depend on the GPU's clock.  By CTAs of 256 particles the smaller takes 0.22 of the larger,
by CTAs of 32 a third."""

import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def sweeps_seconds(n, sweeps=1000):
    import frictionqpotspringblock_gb300 as fqsb

    s = fqsb.Line1d.System_Cuspy_Laplace_Nopassing(mu=1.0, k_interactions=1.0, k_frame=1.0 / n, shape=[n], seed=0,
                                                   distribution="weibull", parameters=[2.0, 1.0, 1e-5], offset=-50.0,
                                                   nchunk=100)
    u0 = np.random.default_rng(1).normal(0.0, 0.3, n)
    best = np.inf
    for _ in range(4):
        s.u = u0
        s.u_frame = 0.5
        t0 = time.perf_counter()
        s.minimise(tol=1e-12, max_iter=sweeps, max_iter_is_error=False)
        best = min(best, time.perf_counter() - t0)
    return best


def test_launch_shape():
    ratio = sweeps_seconds(2 ** 17) / sweeps_seconds(2 ** 20)
    assert ratio < 0.27, ratio
