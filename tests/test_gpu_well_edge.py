"""Positions within a few units of the last place of a yield position: the well test of a Cuspy step
(from the well's centre and half width, then exactly) picks the well of the CPU oracle."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape, offset", [([1500], -100.0), ([64], -3000.0), ([20011], -100.0), ([33, 67], -100.0)])
def test_well_at_its_edges(shape, offset):
    import frictionqpotspringblock_gb300 as fqsb
    from oracle import oracle as O

    n = int(np.prod(shape))
    par = dict(m=1.0, eta=0.1, mu=1.0, k_interactions=1.0, k_frame=1.0 / n, dt=0.1, shape=shape, seed=5,
               distribution="weibull", parameters=[2.0, 1.0, 1e-5], offset=offset, nchunk=500)
    grid = len(shape) == 2
    gpu = (fqsb.Line2d if grid else fqsb.Line1d).System_Cuspy_Laplace(**par)
    ref = (O.line2d if grid else O.line1d)(**par, sum_mode=O.SUM_PAIRWISE, math_mode=O.MATH_PORTABLE)
    rng = np.random.default_rng(1)
    y = gpu.chunk.data.reshape(n, -1)[np.arange(n), 80 + np.arange(n) % 40].reshape(shape)
    ulp = np.spacing(np.abs(y))
    u = y + rng.integers(-4, 5, shape) * ulp
    v = rng.integers(-40, 41, shape) * ulp / 0.1
    a = np.zeros(shape)
    for s in (gpu, ref):
        s.u, s.v, s.a = u, v, a
    for _ in range(3):
        gpu.timeSteps(1)
        ref.timeSteps(1)
        assert np.array_equal(gpu.chunk.index_at_align, ref.chunk.index_at_align)
        assert np.array_equal(gpu.u, ref.u) and np.array_equal(gpu.a, ref.a)
        u, v = gpu.u, rng.integers(-40, 41, shape) * ulp / 0.1
        for s in (gpu, ref):
            s.v, s.a = v, a
