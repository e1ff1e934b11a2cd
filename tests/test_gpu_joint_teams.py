"""The joint multi-band swarm runs a task on a cluster of four blocks, on one
block with an SM to itself, or on one of two blocks an SM, by the size of the
batch.  Sources whose bands sit at the edges of the split of a particle's
observations over its lanes (2 to 8), with two to six bands, and one whose
residuals FP32 cannot square, are fitted in a batch of each form; every output
has to be the same bit for bit."""
import numpy as np
import pytest

from lightcurve_fitting_gb300 import abi, synth

pytestmark = pytest.mark.gpu

EDGES = [(1, 2), (7, 8, 9), (3, 4, 5), (15, 16, 17), (31, 30, 33), (5, 6, 7, 8, 9, 10), (64, 3), (20, 0, 12),
         (63, 65, 2, 40)]


def _batch(layouts, seed, huge=()):
    rng = np.random.default_rng(seed)
    t, f, e, bo, so = [], [], [], [0], [0]
    for k, ns in enumerate(layouts):
        peak = rng.uniform(20, 60)
        for b, n in enumerate(ns):
            x = np.sort(rng.uniform(0, 150, n))
            y = 100 * np.exp(-0.5 * ((x - peak - 3 * b) / rng.uniform(8, 25)) ** 2) + rng.normal(0, 2, n)
            s = np.full(n, 2.0)
            if k in huge and n > 1:
                y[0], s[0] = -1e18, 1.0
            t.append(x)
            f.append(y)
            e.append(s)
            bo.append(bo[-1] + n)
        so.append(so[-1] + len(ns))
    return synth.PhotometryBatch(np.concatenate(t), np.concatenate(f), np.concatenate(e), np.asarray(bo, np.int64),
                                 np.asarray(so, np.int32), np.zeros(len(layouts), np.int32), "edges")


@pytest.fixture(scope="module")
def ctx():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from lightcurve_fitting_gb300 import build
    build.build()
    from lightcurve_fitting_gb300.lib import Context
    c = Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("padding", [60, 200])
def test_joint_fit_does_not_depend_on_the_team(ctx, padding):
    layouts = EDGES + [(12, 13, 14)]
    huge = (len(layouts) - 1,)
    kw = dict(fit_all_models=False, method=abi.METHOD_LAPLACE, run_multi_bazin=False, joint_multiband=True)
    few = ctx.fit_batch(_batch(layouts, 3, huge), **kw)
    # the same draws make the same first sources
    many = ctx.fit_batch(_batch(layouts + [(8, 8)] * padding, 3, huge), **kw)
    n = sum(len(ns) for ns in layouts)
    for name, _ in abi.FitOutputs._fields_:
        a, b = getattr(few, name), getattr(many, name)[:n]
        assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f"), name
