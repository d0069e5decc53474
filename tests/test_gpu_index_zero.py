"""Window moves down to the wells of index -1 and -2 (a particle pushed back below its first yield position): by the
positions' setter and inside runs, on every path.  Against the CPU oracle."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def both(n, **kw):
    import frictionqpotspringblock_gb300 as fqsb
    from oracle import oracle as O

    par = dict(m=1.0, eta=0.1, mu=1.0, k_interactions=0.1, k_frame=0.1, dt=0.1, shape=[n], seed=3, distribution="delta",
               parameters=[1.0], offset=-5.0, nchunk=40)
    par.update(kw)
    gpu = fqsb.Line1d.System_Cuspy_Laplace(**par)
    ref = O.line1d(**par, sum_mode=O.SUM_PAIRWISE, math_mode=O.MATH_PORTABLE)
    return gpu, ref


def same(gpu, ref):
    for name in ("u", "v", "a", "f", "f_potential"):
        assert np.array_equal(getattr(gpu, name), getattr(ref, name)), name
    assert np.array_equal(gpu.chunk.index_at_align, ref.chunk.index_at_align)
    assert np.array_equal(gpu.chunk.start, ref.chunk.start)


# the first yield position is -4: the well of index i is [i - 4, i - 3)
@pytest.mark.parametrize("index", [-4, -3, -2, -1, 0, 1])
def test_set_u(index):
    gpu, ref = both(64)
    for start in range(-8, 3):
        for i in (60, start + 35, index):
            # i = start + 35 is at least 6 below the window before, and moves it to `start` + 5
            u = np.full(64, i - 3.5)
            gpu.u = u
            ref.u = u
            same(gpu, ref)


@pytest.mark.parametrize("path", ["cluster", "run", "steps"])
@pytest.mark.parametrize("distribution, parameters", [("delta", [1.0]), ("weibull", [2.0, 1.0, 1e-5])])
def test_inside_runs(monkeypatch, path, distribution, parameters):
    if path != "cluster":
        monkeypatch.setenv("FQSB_NO_SMALL", "1")
    if path == "steps":
        monkeypatch.setenv("FQSB_NO_RUN", "1")
    n = 700
    gpu, ref = both(n, distribution=distribution, parameters=parameters)
    rng = np.random.default_rng(1)
    for s in (gpu, ref):
        s.u = np.full(n, 45.0)
        s.u = np.full(n, 20.0)
    u = rng.uniform(-4.0, 3.0, n)
    v = rng.uniform(-6.0, 6.0, n)
    for s in (gpu, ref):
        s.u, s.v = u, v
    for k in (1, 2, 40):
        for s in (gpu, ref):
            s.timeSteps(k)
        same(gpu, ref)
    for s in (gpu, ref):
        s.v = -v
        s.flowSteps(60, -1.0)
    same(gpu, ref)
    kw = dict(max_iter=100, max_iter_is_error=False)
    assert gpu.minimise(time_activity=True, **kw) == ref.minimise(time_activity=True, **kw)
    same(gpu, ref)
