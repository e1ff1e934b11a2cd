"""The rules that pick how a band is fitted by the size of its batch: a warp or
eight lanes a band in the polish, four warps or one in the SVI, a block or a
warp a swarm.  Bands whose lengths sit at the edges of those rules are fitted
in a small batch, in one padded with short sources past every batch-size rule,
and one by one; every output has to be the same bit for bit (each rule keeps a
band's order of summation)."""
import numpy as np
import pytest

from lightcurve_fitting_gb300 import abi, synth

pytestmark = pytest.mark.gpu

EDGES = [(1, 7, 8), (9, 31, 32), (33, 63, 64), (65, 95, 96), (97, 127, 128), (129, 160, 255), (256, 257, 300),
         (31, 128, 129), (5, 6, 256), (2, 3, 4)]
PADDING = 4200  # sources: 12,630 bands with the edges


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


def _cut(layout, seed):
    """Sources with the given numbers of points a band."""
    layout = np.asarray(layout)
    base = synth.config_uneven(len(layout), seed=seed)
    big = synth.generate(len(layout), np.maximum(layout, 8) * 3, base.generator, seed=seed, t_span=300.0, drop_nights=0.2)
    t, f, e, bo = [], [], [], [0]
    for s, ns in enumerate(layout):
        for (tt, ff, ee), n in zip(big.bands_of(s), ns):
            n = min(int(n), tt.size)
            keep = np.sort(np.random.default_rng(seed + s).permutation(tt.size)[:n])
            t.append(tt[keep])
            f.append(ff[keep])
            e.append(ee[keep])
            bo.append(bo[-1] + n)
    so = (np.arange(len(layout) + 1) * 3).astype(np.int32)
    return synth.PhotometryBatch(np.concatenate(t), np.concatenate(f), np.concatenate(e), np.asarray(bo, np.int64), so,
                                 big.generator, "edges")


def _join(a, b):
    return synth.PhotometryBatch(np.concatenate([a.times, b.times]), np.concatenate([a.flux, b.flux]),
                                 np.concatenate([a.flux_err, b.flux_err]),
                                 np.concatenate([a.band_obs_offsets, a.n_obs + b.band_obs_offsets[1:]]),
                                 np.concatenate([a.source_band_offsets, a.n_bands + b.source_band_offsets[1:]]).astype(np.int32),
                                 np.concatenate([a.generator, b.generator]), "joined")


@pytest.mark.parametrize("method", [abi.METHOD_SVI, abi.METHOD_LAPLACE])
@pytest.mark.parametrize("mode", ["all", "gated", "metzger"])
def test_a_band_is_fitted_alike_in_any_batch(ctx, method, mode):
    kw = dict(fit_all_models=mode == "all", method=method, forced_model=7 if mode == "metzger" else -1)
    edge = _cut(EDGES, seed=77)
    pad = _cut(np.full((PADDING, 3), 5), seed=78)
    small = ctx.fit_batch(edge, **kw)
    large = ctx.fit_batch(_join(edge, pad), **kw)
    assert np.sum(small.model >= 0) == edge.n_bands
    for name, _ in abi.FitOutputs._fields_:
        a, b = getattr(small, name), getattr(large, name)[:edge.n_bands]
        assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f"), name
    for s in range(edge.n_sources):
        one = ctx.fit_batch(edge.subset([s]), **kw)
        for name, _ in abi.FitOutputs._fields_:
            a, b = getattr(small, name)[3 * s:3 * s + 3], getattr(one, name)
            assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f"), (s, name)
