"""A swarm run by a whole block ends where a warp's does.

Bands of 32 points or more go to blocks in a batch that has at most 64 of
them, and none do in a batch with more than 300 bands of 512 points or more.
1,000 uneven sources and three long ones (several chunks of a block's terms;
bands beyond a warp's and beyond a block's staging memory) are fitted both
ways: by 21 sources at a time, and all at once beside such long bands.  Every
swarm's row and every output has to be the same bit for bit: the block adds a
warp's terms in a warp's order, and both compile the same expressions.  A last
bit that moves shows in about one swarm of 100,000, hence the number."""
import numpy as np
import pytest

from lightcurve_fitting_gb300 import abi, synth

pytestmark = pytest.mark.gpu

GROUP = 21  # sources: 63 bands


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


def _long(layout, seed):
    """Sources with the given numbers of points a band (noise drops some of a
    generated band's points, so from bands of several times as many)."""
    layout = np.asarray(layout)
    pool = synth.generate(len(layout), 6 * layout, np.zeros(len(layout), np.int64), seed=seed, t_span=1000.0,
                          drop_nights=0.0, amp_lo=1.0e5, amp_hi=1.0e6)
    rng = np.random.default_rng(seed)
    cut = [pool.band_obs_offsets[b] + np.sort(rng.choice(c, n, replace=False))
           for b, (c, n) in enumerate(zip(pool.band_counts(), layout.reshape(-1)))]
    i = np.concatenate(cut)
    return synth.PhotometryBatch(pool.times[i], pool.flux[i], pool.flux_err[i],
                                 np.concatenate([[0], np.cumsum(layout)]), pool.source_band_offsets, pool.generator, "long")


def _join(*parts):
    bo, so = [np.zeros(1, np.int64)], [np.zeros(1, np.int64)]
    for p in parts:
        bo.append(bo[-1][-1] + p.band_obs_offsets[1:])
        so.append(so[-1][-1] + p.source_band_offsets[1:])
    cat = lambda name: np.concatenate([getattr(p, name) for p in parts])  # noqa: E731
    return synth.PhotometryBatch(cat("times"), cat("flux"), cat("flux_err"), np.concatenate(bo),
                                 np.concatenate(so).astype(np.int32), cat("generator"), "joined")


def _fit(ctx, batch, kw):
    res = ctx.fit_batch(batch, **kw)
    out = {name: getattr(res, name) for name, _ in abi.FitOutputs._fields_}
    rows, nb = ctx.swarm_results(batch.n_bands), batch.n_bands
    out["swarms"] = rows[:24 * nb].reshape(nb, 24, -1)  # (model, restart)
    out["t0 search"] = rows[24 * nb:32 * nb].reshape(nb, 8, -1)
    out["MultiBazin"] = rows[32 * nb:].reshape(nb, 12, -1)
    return out


@pytest.mark.parametrize("candidate", [0, 1, 2])
@pytest.mark.parametrize("mode", ["all", "gated", "villar"])
def test_block_and_warp_swarms_agree(ctx, mode, candidate):
    kw = dict(fit_all_models=mode == "all", method=abi.METHOD_SVI, forced_model=1 if mode == "villar" else -1)
    field = synth.config_uneven(1000, seed=1000 + 10 * candidate, max_count=500)
    dense = _long([(3300, 1500, 700), (513, 512, 511), (160, 129, 128)], seed=3)
    filler = _long(np.full((101, 3), 512), seed=4)
    n = field.n_bands + dense.n_bands
    ctx.set_autotune(1, candidate)
    try:
        warps = _fit(ctx, _join(field, dense, filler), kw)
        parts = [_fit(ctx, field.subset(range(s, min(s + GROUP, field.n_sources))), kw)
                 for s in range(0, field.n_sources, GROUP)]
        parts.append(_fit(ctx, dense, kw))
    finally:
        ctx.set_autotune(1, -1)
    for name in parts[0]:
        a, b = np.concatenate([p[name] for p in parts]), warps[name][:n]
        assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f"), name
