"""launch_batch_svi_fit with upper limits whose flux is NaN: each adds
ln 1e-300 to a sample's log-likelihood (log_normal_cdf's floor: the maximum of
a NaN probability and 1e-300 is 1e-300, cuda/models_device.h).  One step's ELBO
is then that of the band without those limits plus ln 1e-300 a limit; the two
add the same other terms in another order (60 terms of 1e2 at most: 1e-11)."""
import numpy as np
import pytest

from lightcurve_fitting_gb300 import abi, synth

pytestmark = pytest.mark.gpu

CENTRE = [[0.3, 0.0, 40.0, 1.6, 3.4, -2.0], [0.2, 0.005, 2.9, 40.0, 1.4, 3.5, -2.0], [0.3, 0.0, 40.0, 1.5, 3.3, 1.67, -2.0],
          [0.6, 30.0, 2.4, 0.0, -2.0], [0.6, 30.0, 3.0, 2.3, -2.0], [0.4, 30.0, 0.4, 2.6, -2.0]]


@pytest.fixture(scope="module")
def L():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from lightcurve_fitting_gb300 import build
    build.build()
    from lightcurve_fitting_gb300.lib import load
    return load()


def _elbo(L, m, t, f, var, up, uf):
    import torch
    dev = lambda a, dt: torch.tensor(np.asarray(a, dt), device="cuda")  # noqa: E731
    args = [dev(t, np.float64), dev(f, np.float64), dev(var, np.float64), dev(up, np.int32), dev(uf, np.float64),
            dev([0, len(t)], np.int32), dev(CENTRE[m], np.float64), dev([m], np.int32), dev([abi.N_PARAMS[m]], np.int32),
            dev([abi.SE_IDX[m]], np.int32), dev(CENTRE[m], np.float64), dev(np.ones(len(CENTRE[m])), np.float64)]
    out = [torch.zeros(7, dtype=torch.float64, device="cuda") for _ in range(2)]
    elbo = torch.zeros(1, dtype=torch.float64, device="cuda")
    L.launch_batch_svi_fit(*[a.data_ptr() for a in args + out], elbo.data_ptr(), 1, len(CENTRE[m]), 1, 4, 0.01, 1, 256)
    torch.cuda.synchronize()
    return float(elbo)


@pytest.mark.parametrize("m", range(6))  # the afterglow ELBO here is too large to show a term of 700
def test_nan_upper_limits_add_the_floor(L, m):
    t, f, e = max(synth.config_gradient(1, seed=5).bands_of(0), key=lambda b: b[0].size)
    f, e = f / f.max(), e / f.max()
    var, up, uf = e * e + 1e-4, (f / e < 3.0).astype(np.int32), 3.0 * e
    nan = np.arange(4, t.size, 9)
    up[nan], uf[nan] = 1, np.nan
    keep = np.setdiff1d(np.arange(t.size), nan)
    want = _elbo(L, m, t[keep], f[keep], var[keep], up[keep], uf[keep]) + nan.size * np.log(1e-300)
    got = _elbo(L, m, t, f, var, up, uf)
    assert np.isfinite(want)
    assert abs(got - want) <= 1e-11 * abs(want)
