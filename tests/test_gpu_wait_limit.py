"""A wait of the run kernel's CTAs for one another that runs out (csrc/fqsb_run.cu): a healthy run is given a limit
shorter than one of its steps.  The run ends with the timeout status, and the handle can be used again."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 2 ** 22


def ring():
    import frictionqpotspringblock_gb300 as fqsb

    # (the Smooth potential: a step takes about a millisecond)
    return fqsb.Line1d.System_Smooth_Laplace(m=1.0, eta=0.1, mu=1.0, k_interactions=1.0, k_frame=1.0 / N, dt=0.1, shape=[N],
                                             seed=3, distribution="weibull", parameters=[2.0, 1.0, 1e-5], offset=-5.0,
                                             nchunk=34)


def grid():
    import frictionqpotspringblock_gb300 as fqsb

    return fqsb.Line2d.System_Cuspy_Laplace(m=1.0, eta=0.2, mu=1.0, k_interactions=1.0, k_frame=0.01, dt=0.1,
                                            shape=[4096, 2048], seed=3, distribution="weibull",
                                            parameters=[2.0, 1.0, 1e-5], offset=-5.0, nchunk=34)


@pytest.mark.parametrize("make", [ring, grid])
def test_wait_runs_out(make):
    from frictionqpotspringblock_gb300 import _capi

    def limit(s, ns):
        assert _capi.lib().fqsb_set_wait_limit(s._h, ctypes.c_uint64(ns)) == _capi.OK

    s = make()
    u0 = np.random.default_rng(1).normal(0.0, 0.1, s.size).reshape(s.shape)
    zero = np.zeros(s.shape)

    def run():
        s.u, s.v, s.a = u0, zero, zero
        s.u_frame, s.inc = 0.0, 0
        s.flowSteps(6, 0.5)
        s.minimise(max_iter=4, max_iter_is_error=False)
        return s.u, s.v, s.chunk.index_at_align, s.inc

    expect = run()
    for _ in range(2):
        s.u = u0
        limit(s, 1)
        with pytest.raises(RuntimeError, match="ran out"):
            s.flowSteps(300, 0.5)
        limit(s, 5 * 10 ** 9)
        for a, b in zip(expect, run()):
            assert np.array_equal(a, b)
