"""The SVI's MetzgerKN predictions and tangents (a warp a sample) through
lcf_svi_elbo_grad, which runs the same function: bands of one observation to
more than a warp takes at once, with t0 at the places where the evaluation
changes its form (before the band, inside it, an observation at phase 0 or
before the grid's first point, at and past the last observation).

Against the FP64 oracle: the ELBO to 1e-5 of max(|ELBO|, 1) (FP32 terms), and,
for t0 inside the band's span, the gradient's median error to 1e-4 (the
reference's model gradient is a forward difference with step 1e-5)."""
import numpy as np
import pytest

from lightcurve_fitting_gb300 import abi

pytestmark = pytest.mark.gpu


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


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 31, 32, 33, 70])
def test_elbo_of_the_warp_form(ctx, oracle, n):
    rng = np.random.default_rng(50 + n)
    # times that FP32 holds exactly, so that both sides see the same phases
    t = 8.0 + np.sort(rng.choice(64 * 40, n, replace=False)) / 64.0
    f = np.exp(-0.08 * (t - t[0])) * (1.0 + 0.05 * rng.standard_normal(n))
    f /= f.max()
    e = np.full(n, 0.05)
    band = oracle.Band(t, f, e)
    band.up = np.zeros_like(band.up)
    last = t[-1]
    inside = [t[0] - 4.0, t[0] - 1.5, 0.5 * (t[0] + last) - 1.0 / 128]
    edges = [t[0], t[0] - 1.0 / 256, t[-1] - 1.0 / 256, last, last + 3.0]
    errs, compared = [], 0
    for k, t0 in enumerate(inside + edges):
        mu = np.array([-1.8, -1.0, 0.4, t0, -2.0])
        vp = np.concatenate([mu, np.full(5, -3.0)])
        init, eps = mu + 0.1, np.zeros((1, 5))
        want, grad, flags = oracle.svi_elbo_grad(7, band, init, vp, eps)
        got, g, fl = ctx.svi_elbo_grad(7, band.t, band.f, band.var, band.up, band.uf, init, vp[None], eps[None])
        assert fl[0] == flags, (n, k)
        assert abs(got[0] - want) <= 1e-5 * max(abs(want), 1.0), (n, k, got[0], want)
        assert np.all(np.isfinite(g))
        if k < len(inside) and flags == 0:
            errs.append(np.max(np.abs(g[0] - grad)) / np.max(np.abs(grad)))
            compared += 1
    assert compared == 0 or np.median(errs) < 1e-4, errs
