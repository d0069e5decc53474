"""Forces at the lower end of binary64.  A product by a power of two is exact only where it is not subnormal: the
fused force sums (csrc/fqsb_device.cuh, scale_add) have to round there as product and sum do.  A particle that relaxes
towards a well centred at 0 gets there.  Bit for bit against the CPU oracle."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["ring", "grid", "particles", "semismooth", "ensemble of one step", "one step grid"])
@pytest.mark.parametrize("scale", [-1074, -1066, -1022, -1000, -960])
def test_subnormal_products(monkeypatch, kind, scale):
    import frictionqpotspringblock_gb300 as fqsb
    from oracle import oracle as O

    monkeypatch.setenv("FQSB_NO_SMALL", "1")
    exact = dict(sum_mode=O.SUM_PAIRWISE, math_mode=O.MATH_PORTABLE)
    shape = [70, 61] if "grid" in kind else [5003]
    par = dict(m=1.0, eta=0.5, mu=1.0, k_frame=0.25, dt=0.25, shape=shape, seed=3, distribution="delta",
               parameters=[1.0], offset=-49.5, nchunk=100)
    if "grid" in kind:
        gpu = fqsb.Line2d.System_Cuspy_Laplace(k_interactions=0.25, **par)
        ref = O.line2d(k_interactions=0.25, **par, **exact)
    elif kind == "particles":
        gpu = fqsb.Particles.System_Cuspy(**par)
        ref = O.particles("Cuspy", **par, **exact)
    elif kind == "semismooth":
        gpu = fqsb.Line1d.System_SemiSmooth_Laplace(kappa=0.5, k_interactions=0.25, **par)
        ref = O.line1d("SemiSmooth", kappa=0.5, k_interactions=0.25, **par, **exact)
    else:
        gpu = fqsb.Line1d.System_Cuspy_Laplace(k_interactions=0.25, **par)
        ref = O.line1d(k_interactions=0.25, **par, **exact)
    rng = np.random.default_rng(scale + 2000)
    u = np.ldexp(rng.integers(-200, 200, shape).astype(np.float64), scale)
    v = np.ldexp(rng.integers(-200, 200, shape).astype(np.float64), scale)
    gpu.u, gpu.v = u, v
    ref.u, ref.v = u, v
    for steps in (1, 1, 6) if "step" in kind else (2, 6):
        gpu.timeSteps(steps)
        ref.timeSteps(steps)
        for name in ("u", "v", "a"):
            g, r = getattr(gpu, name), getattr(ref, name)
            assert np.array_equal(g.view(np.int64), np.asarray(r).reshape(g.shape).view(np.int64)), (name, np.sum(g != r))
