"""Thermal forcing at the limits of its plans (csrc/fqsb_thermal.cu): the largest numbers of steps, and plans of
few steps over many particles."""

import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def both(n, **kw):
    import frictionqpotspringblock_gb300 as fqsb
    from oracle import oracle as O

    rng = np.random.default_rng(n)
    par = dict(m=1.0, eta=0.3, mu=1.0, k_interactions=1.0, k_frame=0.1, dt=0.1, mean=0.05, stddev=0.4, seed_forcing=9,
               dinc_init=rng.integers(0, 40, n), dinc=rng.integers(1, 40, n), shape=[n], seed=4,
               distribution="weibull", parameters=[2.0, 1.0, 1e-5], offset=-20.0, nchunk=45)
    par.update(kw)
    gpu = fqsb.Line1d.System_Cuspy_Laplace_RandomForcing(**par)
    ref = O.line1d_random_forcing(**par, sum_mode=O.SUM_PAIRWISE, math_mode=O.MATH_PORTABLE)
    return gpu, ref


def same(gpu, ref):
    for name in ("u", "v", "a", "f", "f_frame"):
        assert np.array_equal(getattr(gpu, name), getattr(ref, name)), name
    assert np.array_equal(gpu.external.f_thermal, ref.f_thermal)
    assert np.array_equal(gpu.external.next, ref.thermal_next)
    assert gpu.external.state == ref.thermal_state
    assert np.array_equal(gpu.chunk.index_at_align, ref.chunk.index_at_align)
    assert gpu.inc == ref.inc


@pytest.mark.parametrize("path", ["cluster", "graph"])
@pytest.mark.parametrize("max_iter", [2 ** 63 - 1, 2 ** 63 - 200, 4096, 4095])
def test_many_steps_allowed(monkeypatch, path, max_iter):
    """The number of launches for the steps allowed does not overflow."""
    if path == "graph":
        monkeypatch.setenv("FQSB_NO_SMALL", "1")
    gpu, ref = both(1000, stddev=0.05)
    assert gpu.timeStepsUntilEvent(max_iter=max_iter) == ref.timeStepsUntilEvent(max_iter=min(max_iter, 10 ** 9))
    same(gpu, ref)


@pytest.mark.parametrize("n", [8191, 8193, 2 ** 19 + 1])
def test_blocks_of_particles(monkeypatch, n):
    """The draws are counted and listed by blocks of 8192 particles: their edges, and many of them."""
    gpu, ref = both(n, dinc=np.random.default_rng(n).choice([1, 3, 50, 100000], n, p=[0.05, 0.05, 0.4, 0.5]))
    for k in (1, 33) if n > 100000 else (1, 300, 2):
        gpu.flowSteps(k, 1.0)
        ref.flowSteps(k, 1.0)
        same(gpu, ref)


def test_one_step_plans():
    """Above 2^21 particles a plan holds one step, by the step kernel of two particles per thread."""
    n = 2 ** 21 + 77
    gpu, ref = both(n, dinc_init=np.random.default_rng(1).integers(0, 4, n), dinc=np.random.default_rng(2).integers(4, 90, n),
                    nchunk=34)
    for k in (1, 5):
        gpu.flowSteps(k, 1.0)
        ref.flowSteps(k, 1.0)
        same(gpu, ref)


def step_seconds(n, steps=50):
    gpu = both_gpu(n)
    gpu.flowSteps(steps, 1e-3)
    best = np.inf
    for _ in range(4):
        t0 = time.perf_counter()
        gpu.flowSteps(steps, 1e-3)
        best = min(best, time.perf_counter() - t0)
    return best / steps


def both_gpu(n, **kw):
    import frictionqpotspringblock_gb300 as fqsb

    par = dict(m=1.0, eta=0.1, mu=1.0, k_interactions=1.0, k_frame=1.0 / n, dt=0.1, mean=0.0, stddev=0.05, seed_forcing=9,
               dinc_init=np.random.default_rng(n).integers(0, 100, n), dinc=np.full(n, 100), shape=[n], seed=4,
               distribution="weibull", parameters=[2.0, 1.0, 1e-5], offset=-20.0, nchunk=40)
    par.update(kw)
    return fqsb.Line1d.System_Cuspy_Laplace_RandomForcing(**par)


def test_large_systems_fill_the_gpu():
    """Four times the particles take about four times as long (one CTA per planned step: twelve times)."""
    ratio = step_seconds(2 ** 22) / step_seconds(2 ** 20)
    assert ratio < 6.5, ratio


DRIVEN = dict(k_frame=0.5, eta=0.5, nchunk=40)


@pytest.mark.parametrize("n", [40, 5003, 40001])
def test_plan_outlives_window_moves(monkeypatch, n):
    """A launch of the run kernel ends at every step in which windows move; the plan goes on behind it, over its own
    end and from run to run."""
    monkeypatch.setenv("FQSB_NO_SMALL", "1")
    gpu, ref = both(n, **DRIVEN)
    for k in (1, 254, 3, 300) if n < 10000 else (1, 120, 3):
        gpu.flowSteps(k, 2.0)
        ref.flowSteps(k, 2.0)
        same(gpu, ref)
    assert np.array_equal(gpu.chunk.start, ref.chunk.start) and np.max(ref.chunk.start) > 0
    gpu.external.state = ref.thermal_state = 0x9E3779B97F4A7C15
    gpu.flowSteps(20, 2.0)
    ref.flowSteps(20, 2.0)
    same(gpu, ref)


def driven_seconds(s, steps=300):
    s.flowSteps(steps, 2.0)
    best = np.inf
    for _ in range(3):
        t0 = time.perf_counter()
        s.flowSteps(steps, 2.0)
        best = min(best, time.perf_counter() - t0)
    return best


def test_window_moves_plan_once():
    """Where windows move in most steps, thermal forcing costs less than the step itself (with a plan for every launch
    it cost one and a half steps)."""
    import frictionqpotspringblock_gb300 as fqsb

    n = 65536
    athermal = fqsb.Line1d.System_Cuspy_Laplace(m=1.0, mu=1.0, k_interactions=1.0, dt=0.1, shape=[n], seed=4,
                                                distribution="weibull", parameters=[2.0, 1.0, 1e-5], offset=-20.0, **DRIVEN)
    ratio = driven_seconds(both_gpu(n, **DRIVEN)) / driven_seconds(athermal)
    assert ratio < 2.0, ratio
