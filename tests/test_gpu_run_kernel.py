"""Resident run kernel (csrc/fqsb_run.cu) at the edges of its work split -- one strip, ragged strips, the
sizes where strips get longer and nodes larger -- and of its runs: one step, a stop that drops the step
taken after it, steps that end a launch because windows must move.  Bit for bit against the CPU oracle."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("u", "v", "a", "f", "f_frame")


def both(monkeypatch, n, **kw):
    import frictionqpotspringblock_gb300 as fqsb
    from oracle import oracle as O

    par = dict(m=1.0, eta=0.1, mu=1.0, k_interactions=1.0, k_frame=1.0 / n, dt=0.1, shape=[n], seed=11,
               distribution="weibull", parameters=[2.0, 1.0, 1e-5], offset=-20.0, nchunk=60)
    par.update(kw)
    monkeypatch.setenv("FQSB_NO_SMALL", "1")
    gpu = fqsb.Line1d.System_Cuspy_Laplace(**par)
    ref = O.line1d(**par, sum_mode=O.SUM_PAIRWISE, math_mode=O.MATH_PORTABLE)
    u = np.random.default_rng(n).normal(0.0, 0.3, n)
    gpu.u = u
    ref.u = u
    return gpu, ref


def same(gpu, ref):
    for name in FIELDS:
        assert np.array_equal(getattr(gpu, name), getattr(ref, name)), name
    assert np.array_equal(gpu.chunk.index_at_align, ref.chunk.index_at_align)
    assert np.array_equal(gpu.chunk.start, ref.chunk.start)
    assert gpu.inc == ref.inc and gpu.u_frame == ref.u_frame


# 32 * 151 * 28 = 135296 particles fill the strips of 32 on a GPU of 152 SMs; 2 and 8 times as many those of 64, 256
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 1023, 4833, 38913, 135296, 135297, 270593, 1082369])
def test_strips(monkeypatch, n):
    gpu, ref = both(monkeypatch, n)
    for steps in (1, 2, 7) if n < 300000 else (1, 3):
        gpu.timeSteps(steps)
        ref.timeSteps(steps)
        same(gpu, ref)
    for max_iter in (1, 4) if n < 300000 else (3,):
        kw = dict(max_iter=max_iter, max_iter_is_error=False)
        assert gpu.minimise(**kw) == ref.minimise(**kw)
        assert gpu.minimise(time_activity=True, **kw) == ref.minimise(time_activity=True, **kw)
        same(gpu, ref)
    assert gpu.residual == ref.residual


@pytest.mark.parametrize("n", [40, 3000, 40000])
@pytest.mark.parametrize("activity", [False, True])
def test_stop_and_window_moves(monkeypatch, n, activity):
    gpu, ref = both(monkeypatch, n, nchunk=40, k_frame=0.5, eta=0.5)
    gpu.flowSteps(150, 2.0)
    ref.flowSteps(150, 2.0)
    same(gpu, ref)
    assert np.max(gpu.chunk.start) > 0
    assert gpu.minimise(time_activity=activity) == ref.minimise(time_activity=activity) == 0
    same(gpu, ref)
    gpu.u_frame = gpu.u_frame + 1.0
    ref.u_frame = ref.u_frame + 1.0
    i = ref.chunk.index_at_align.copy()
    kw = dict(i_n=i, A_truncate=max(1, n // 8))
    assert gpu.minimise_truncate(**kw) == ref.minimise_truncate(**kw)
    same(gpu, ref)
    gpu.u_frame = gpu.u_frame + 0.1
    ref.u_frame = ref.u_frame + 0.1
    assert gpu.timeStepsUntilEvent() == ref.timeStepsUntilEvent()
    same(gpu, ref)
