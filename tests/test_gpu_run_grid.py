"""Laplace2d systems on the resident run kernel (csrc/fqsb_run.cu): strips of the flat index of grids with one row, one
column, fewer columns than a strip and many more, ragged last strips; single steps and runs (the positions
that a step leaves for the next), stops and window moves.  Bit for bit against the CPU oracle."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("u", "v", "a", "f", "f_frame", "f_interactions")


def both(shape, **kw):
    import frictionqpotspringblock_gb300 as fqsb
    from oracle import oracle as O

    n = int(np.prod(shape))
    par = dict(m=1.0, eta=0.1, mu=1.0, k_interactions=1.0, k_frame=1.0 / n, dt=0.1, shape=list(shape), seed=23,
               distribution="weibull", parameters=[2.0, 1.0, 1e-5], offset=-20.0, nchunk=60)
    par.update(kw)
    gpu = fqsb.Line2d.System_Cuspy_Laplace(**par)
    ref = O.line2d(**par, sum_mode=O.SUM_PAIRWISE, math_mode=O.MATH_PORTABLE)
    u = np.random.default_rng(n).normal(0.0, 0.3, gpu.u.shape)
    gpu.u = u
    ref.u = u.reshape(np.shape(ref.u))
    return gpu, ref


def same(gpu, ref):
    for name in FIELDS:
        assert np.array_equal(np.ravel(getattr(gpu, name)), np.ravel(getattr(ref, name))), name
    assert np.array_equal(np.ravel(gpu.chunk.index_at_align), np.ravel(ref.chunk.index_at_align))
    assert np.array_equal(np.ravel(gpu.chunk.start), np.ravel(ref.chunk.start))
    assert gpu.inc == ref.inc and gpu.u_frame == ref.u_frame


@pytest.mark.parametrize("shape", [(1, 1), (1, 7), (7, 1), (2, 2), (3, 33), (31, 32), (40, 31), (5, 1000), (1000, 5),
                                   (301, 257), (450, 601)])
def test_strips(shape):
    gpu, ref = both(shape)
    for steps in (1, 2, 7):
        gpu.timeSteps(steps)
        ref.timeSteps(steps)
        same(gpu, ref)
    gpu.flowSteps(5, 0.01)
    ref.flowSteps(5, 0.01)
    same(gpu, ref)
    for max_iter in (1, 4):
        kw = dict(max_iter=max_iter, max_iter_is_error=False)
        assert gpu.minimise(**kw) == ref.minimise(**kw)
        assert gpu.minimise(time_activity=True, **kw) == ref.minimise(time_activity=True, **kw)
        same(gpu, ref)
    assert gpu.residual == ref.residual


@pytest.mark.parametrize("shape", [(5, 8), (60, 50), (200, 201)])
@pytest.mark.parametrize("activity", [False, True])
def test_stop_and_window_moves(shape, activity):
    gpu, ref = both(shape, nchunk=40, k_frame=0.5, eta=0.5)
    gpu.flowSteps(150, 2.0)
    ref.flowSteps(150, 2.0)
    same(gpu, ref)
    assert np.max(gpu.chunk.start) > 0
    assert gpu.minimise(time_activity=activity) == ref.minimise(time_activity=activity) == 0
    same(gpu, ref)
    gpu.u_frame = gpu.u_frame + 1.0
    ref.u_frame = ref.u_frame + 1.0
    kw = dict(i_n=ref.chunk.index_at_align.copy(), A_truncate=max(1, int(np.prod(shape)) // 8))
    assert gpu.minimise_truncate(**kw) == ref.minimise_truncate(**kw)
    same(gpu, ref)
    gpu.u_frame = gpu.u_frame + 0.1
    ref.u_frame = ref.u_frame + 0.1
    assert gpu.timeStepsUntilEvent() == ref.timeStepsUntilEvent()
    same(gpu, ref)
