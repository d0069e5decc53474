"""One-cluster run kernel (csrc/fqsb_small.cu) at the edges of its work split -- one CTA, ragged tiles, the sizes
where tiles double and where systems go to the resident run kernel -- and of its runs: one step, stops (each
drops the step taken after it), steps whose windows move.  Bit for bit against the CPU oracle."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("u", "v", "a", "f", "f_frame")


def both(n, pot, **kw):
    import frictionqpotspringblock_gb300 as fqsb
    from oracle import oracle as O

    par = dict(m=1.0, eta=0.1, mu=1.0, k_interactions=1.0, k_frame=1.0 / n, dt=0.1, shape=[n], seed=17,
               distribution="weibull", parameters=[2.0, 1.0, 1e-5], offset=-20.0, nchunk=60)
    par.update(kw)
    cls = {"Cuspy": fqsb.Line1d.System_Cuspy_Laplace, "Smooth": fqsb.Line1d.System_Smooth_Laplace}[pot]
    gpu = cls(**par)
    ref = O.line1d(potential=pot, **par, sum_mode=O.SUM_PAIRWISE, math_mode=O.MATH_PORTABLE)
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


@pytest.mark.parametrize("pot", ["Cuspy", "Smooth"])
@pytest.mark.parametrize("n", [1, 2, 32, 33, 512, 513, 1025, 2048, 2049, 4095, 4096, 4097])
def test_tiles(n, pot):
    gpu, ref = both(n, pot)
    for steps in (1, 2, 3, 130):
        gpu.timeSteps(steps)
        ref.timeSteps(steps)
        same(gpu, ref)
    for max_iter in (1, 2, 70):
        kw = dict(max_iter=max_iter, max_iter_is_error=False)
        assert gpu.minimise(**kw) == ref.minimise(**kw)
        assert gpu.minimise(time_activity=True, **kw) == ref.minimise(time_activity=True, **kw)
        same(gpu, ref)
    assert gpu.residual == ref.residual


@pytest.mark.parametrize("n", [40, 700, 4090])
@pytest.mark.parametrize("activity", [False, True])
def test_stop_and_window_moves(n, activity):
    gpu, ref = both(n, "Cuspy", nchunk=40, k_frame=0.5, eta=0.5)
    gpu.flowSteps(150, 2.0)
    ref.flowSteps(150, 2.0)
    same(gpu, ref)
    assert np.max(gpu.chunk.start) > 0
    assert gpu.minimise(time_activity=activity) == ref.minimise(time_activity=activity) == 0
    same(gpu, ref)
    gpu.u_frame = gpu.u_frame + 1.0
    ref.u_frame = ref.u_frame + 1.0
    kw = dict(i_n=ref.chunk.index_at_align.copy(), A_truncate=max(1, n // 8))
    assert gpu.minimise_truncate(**kw) == ref.minimise_truncate(**kw)
    same(gpu, ref)
    gpu.u_frame = gpu.u_frame + 0.1
    ref.u_frame = ref.u_frame + 0.1
    assert gpu.timeStepsUntilEvent() == ref.timeStepsUntilEvent()
    same(gpu, ref)
