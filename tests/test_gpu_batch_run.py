"""k_batch_run (csrc/fqsb_batch.cu) with one tile per CTA, with several, and the sizes where the batch goes to passes of
k_batch; window moves included.  Bit for bit against passes launched one by one by the host."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COMMON = dict(m=1.0, eta=0.1, mu=1.0, k_interactions=1.0, dt=0.1, distribution="weibull",
              parameters=[2.0, 1.0, 1e-5], offset=-20.0)


# threads 32 x 1 particle: 32 CTAs per SM, 4864 tiles of 32 resident on 152 SMs; 0: the tile left open
@pytest.mark.parametrize("count,hi,threads,ppt", [(1, 16, 32, 1), (30, 5000, 32, 1), (90, 20000, 32, 1),
                                                   (250, 20000, 32, 1), (12, 5000, 0, 0), (90, 20000, 0, 0)])
def test_tiles_per_cta(monkeypatch, count, hi, threads, ppt):
    from frictionqpotspringblock_gb300 import batch as B

    sizes = B.log_uniform_sizes(count, 8, hi, seed=4)
    sizes[0] = 3
    seeds = 1000 + np.arange(len(sizes))
    out = []
    for ng in ("0", "1"):
        monkeypatch.setenv("FQSB_NO_GRAPH", ng)
        b = B.Line1d_System_Cuspy_Laplace(sizes, seeds, 1.0 / sizes, nchunk=100, window=34, threads=threads, ppt=ppt,
                                          **COMMON)
        for cycles, eps in ((1, 1e-3), (2, 0.3)):
            out.append(b.quasistatic(cycles, eps, max_iter=3000))
            out[-1]["u"] = np.concatenate([b.field(j, "u") for j in range(count)])
            out[-1]["i"] = np.concatenate([b.index_at_align(j) for j in range(count)])
        del b
    for a, b in ((out[0], out[2]), (out[1], out[3])):
        for k in ("status", "u", "i"):
            assert np.array_equal(a[k], b[k]), k
        for k in ("u_frame", "f_frame", "S", "inc"):
            # (a realisation that reached max_iter has no outputs of its last cycle)
            assert np.array_equal(a[k][a["status"] == 0], b[k][b["status"] == 0]), k
