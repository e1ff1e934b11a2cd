"""MetzgerKN finalisation of a band with an observation whose time is NaN.  Its
prediction is NaN: the cost is that of a non-finite prediction
(src/parametric.rs:2464-2511: 1e99), the profile scans and the magnitude chi2
leave the observation out (:2716-2726, :4057-4073), and the SVI's ELBO is NaN
rather than that of a finite prediction."""
import numpy as np
import pytest

from lightcurve_fitting_gb300 import abi, synth

pytestmark = pytest.mark.gpu

PARAMS = [-1.75, -1.25, 0.5, -0.5, -2.0]


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


def _band(n):
    """The basic workload's first band: the peak early, so that the last
    observation is neither the peak nor before any t0 of the scans."""
    t, f, e = synth.config_basic(1, seed=3).bands_of(0)[0]
    t, f, e = t[:n].copy(), f[:n].copy(), e[:n].copy()
    f[2] = 2.0 * f.max()
    return t, f, e


def _finalize(ctx, t, f, e, method):
    batch = synth.PhotometryBatch(t, f, e, np.array([0, t.size]), np.array([0, 1], np.int32), np.zeros(1, np.int32), "nan")
    row = np.full((1, 7), np.nan)
    row[0, :5] = PARAMS
    return ctx.finalize_batch(batch, np.array([7], np.int32), row, method=method)


@pytest.mark.parametrize("n", [12, 30])
def test_nan_first_time_is_a_nonfinite_prediction(ctx, n):
    t, f, e = _band(n)
    t[0] = np.nan
    assert _finalize(ctx, t, f, e, abi.METHOD_LAPLACE).svi_elbo[0] == -1e99


@pytest.mark.parametrize("n", [12, 30])
def test_nan_last_time_has_no_prediction(ctx, n):
    t, f, e = _band(n)
    chi2 = _finalize(ctx, t[:-1], f[:-1], e[:-1], abi.METHOD_LAPLACE).mag_chi2[0]
    t[-1] = np.nan
    assert np.isnan(_finalize(ctx, t, f, e, abi.METHOD_SVI).svi_elbo[0])
    # the Laplace means are the parameters given but for the scanned t0
    assert abs(_finalize(ctx, t, f, e, abi.METHOD_LAPLACE).mag_chi2[0] - chi2) <= 1e-12 * abs(chi2)
