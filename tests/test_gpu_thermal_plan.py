"""Planned thermal draws (csrc/fqsb_thermal.cu): runs that end inside, at and beyond the 256 planned steps,
particles that draw every step, now and then, late or never again, chunk windows that move on the way -- on the
one-cluster and on the run-graph path, bit for bit against the CPU oracle."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("u", "v", "a", "f", "f_frame")


@pytest.mark.parametrize("path", ["cluster", "graph"])
@pytest.mark.parametrize("n, steps", [(5, (1, 255, 1)), (33, (256, 257, 3)), (1000, (600, 1)), (40001, (30, 1))])
def test_plan(monkeypatch, path, n, steps):
    import frictionqpotspringblock_gb300 as fqsb
    from oracle import oracle as O

    if path == "graph":
        monkeypatch.setenv("FQSB_NO_SMALL", "1")
    rng = np.random.default_rng(n)
    par = dict(m=1.0, eta=0.3, mu=1.0, k_interactions=1.0, k_frame=0.1, dt=0.1, mean=0.05, stddev=0.4, seed_forcing=9,
               dinc_init=rng.integers(-3, 40, n), dinc=rng.choice([0, 1, 2, 7, 100, 100000], n), shape=[n], seed=4,
               distribution="weibull", parameters=[2.0, 1.0, 1e-5], offset=-20.0, nchunk=45)
    gpu = fqsb.Line1d.System_Cuspy_Laplace_RandomForcing(**par)
    ref = O.line1d_random_forcing(**par, sum_mode=O.SUM_PAIRWISE, math_mode=O.MATH_PORTABLE)
    for k in steps:
        gpu.flowSteps(k, 1.0)
        ref.flowSteps(k, 1.0)
        for name in FIELDS:
            assert np.array_equal(getattr(gpu, name), getattr(ref, name)), (k, name)
        assert np.array_equal(gpu.external.f_thermal, ref.f_thermal)
        assert np.array_equal(gpu.external.next, ref.thermal_next)
        assert gpu.external.state == ref.thermal_state
        assert np.array_equal(gpu.chunk.index_at_align, ref.chunk.index_at_align)
        assert gpu.inc == ref.inc
    assert gpu.timeStepsUntilEvent() == ref.timeStepsUntilEvent()
    assert np.array_equal(gpu.external.f_thermal, ref.f_thermal) and np.array_equal(gpu.u, ref.u)
