"""One kernel per step (FQSB_NO_RUN=1), which GPUs or processes take on which the resident kernels' grids do not fit:
one and two particles per thread, grids, thermal forcing, an ensemble.  Bit for bit against the CPU oracle, or the
resident kernels where those are compared with it elsewhere."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PAR = dict(m=1.0, eta=0.3, mu=1.0, dt=0.1, seed=4, distribution="weibull", parameters=[2.0, 1.0, 1e-5], offset=-20.0,
           nchunk=45)


def systems(kind, shape):
    import frictionqpotspringblock_gb300 as fqsb
    from oracle import oracle as O

    exact = dict(sum_mode=O.SUM_PAIRWISE, math_mode=O.MATH_PORTABLE)
    n = int(np.prod(shape))
    par = dict(PAR, shape=shape, k_frame=0.1)
    th = dict(mean=0.05, stddev=0.3, seed_forcing=9, dinc_init=np.random.default_rng(n).integers(0, 40, n),
              dinc=np.random.default_rng(n).integers(20, 60, n))
    if kind == "ring":
        return fqsb.Line1d.System_Cuspy_Laplace(k_interactions=1.0, **par), O.line1d(k_interactions=1.0, **par, **exact)
    if kind == "grid":
        return fqsb.Line2d.System_Cuspy_Laplace(k_interactions=1.0, **par), O.line2d(k_interactions=1.0, **par, **exact)
    if kind == "thermal ring":
        gpu = fqsb.Line1d.System_Cuspy_Laplace_RandomForcing(k_interactions=1.0, **par, **th)
        ref = O.line1d("Cuspy", k_interactions=1.0, **par, **exact)
    elif kind == "thermal quartic":
        gpu = fqsb.Line1d.System_Cuspy_Quartic_RandomForcing(a1=0.8, a2=0.6, **par, **th)
        ref = O.line1d_quartic(a1=0.8, a2=0.6, **par, **exact)
    else:
        gpu = fqsb.Particles.System_Cuspy_RandomForcing(**par, **th)
        ref = O.particles("Cuspy", **par, **exact)
    O.attach_random_forcing(ref, **th)
    return gpu, ref


def same(gpu, ref):
    for name in ("u", "v", "a", "f", "f_frame"):
        assert np.array_equal(getattr(gpu, name), getattr(ref, name)), name
    assert np.array_equal(gpu.chunk.index_at_align, ref.chunk.index_at_align)
    assert np.array_equal(gpu.chunk.start, ref.chunk.start)
    assert gpu.inc == ref.inc


@pytest.mark.parametrize("kind, shape", [("ring", [1000]), ("ring", [2 ** 18 + 77]), ("grid", [70, 61]),
                                         ("thermal ring", [1000]), ("thermal ring", [2 ** 18 + 77]),
                                         ("thermal quartic", [2 ** 18 + 77]), ("thermal particles", [2 ** 18 + 77])])
def test_parity(monkeypatch, kind, shape):
    monkeypatch.setenv("FQSB_NO_RUN", "1")
    monkeypatch.setenv("FQSB_NO_SMALL", "1")
    gpu, ref = systems(kind, shape)
    steps = 40 if gpu.size > 10000 else 200
    for s in (gpu, ref):
        s.timeSteps(2)
        s.flowSteps(steps, 2.0)
    same(gpu, ref)
    assert np.max(gpu.chunk.start) > 0 or steps == 40
    if "thermal" in kind:
        assert np.array_equal(gpu.external.f_thermal, ref.f_thermal)
        assert gpu.external.state == ref.thermal_state
    else:
        kw = dict(max_iter=60, max_iter_is_error=False)
        assert gpu.minimise(**kw) == ref.minimise(**kw)
        assert gpu.minimise(time_activity=True, **kw) == ref.minimise(time_activity=True, **kw)
        same(gpu, ref)


def test_ensemble(monkeypatch):
    from frictionqpotspringblock_gb300 import batch

    n = np.array([300, 2000, 77, 5000])

    def run():
        b = batch.Line1d_System_Cuspy_Laplace(n, 7 + np.arange(4), 1.0 / n, m=1.0, eta=0.1, mu=1.0, k_interactions=1.0,
                                              dt=0.1, distribution="weibull", parameters=[2.0, 1.0, 1e-5], offset=-5.0,
                                              nchunk=100, window=64)
        out = b.quasistatic(2, 1e-5)
        out["u"] = np.concatenate([b.field(j) for j in range(4)])
        return out

    resident = run()
    monkeypatch.setenv("FQSB_NO_RUN", "1")
    passes = run()
    for name in resident:
        assert np.array_equal(resident[name], passes[name]), name
