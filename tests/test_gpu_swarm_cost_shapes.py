"""launch_batch_pso_cost where its blocks' (particle, slot) layout changes:
one particle, chunk edges (42 and 43, 84 and 85 particles), more particles than
a block has threads, and bands of one observation up to more than a block's
slots.  The costs are FP64 sums in another order than the oracle's, of up to
200 terms: 1e-11 relative, as the other tests of this export hold them."""
import numpy as np
import pytest

from lightcurve_fitting_gb300 import abi, synth

pytestmark = pytest.mark.gpu

BOUNDS = {
    0: ([-1.0, -0.3, 0.0, -2.0, -2.0, -5.0], [1.0, 0.3, 100.0, 5.0, 6.0, 0.0]),
    3: ([-1.0, 0.0, 0.5, -3.0, -5.0], [1.0, 100.0, 4.5, 3.0, 0.0]),
}
LENGTHS = [1, 2, 31, 64, 65, 129, 200, 0]


@pytest.mark.parametrize("m", sorted(BOUNDS))
@pytest.mark.parametrize("particles", [1, 2, 5, 42, 43, 84, 85, 129, 200])
def test_costs_at_the_layout_edges(oracle, m, particles):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    from lightcurve_fitting_gb300.lib import load
    L = load()
    base = synth.generate(len(LENGTHS), np.full((len(LENGTHS), 3), 400), np.zeros(len(LENGTHS), np.int64), seed=5,
                          t_span=150.0, drop_nights=0.0)
    bands = []
    for s, n in enumerate(LENGTHS):
        t, f, e = base.bands_of(s)[0]
        assert t.size >= n
        if n:
            bands.append(oracle.Band(t[:n], f[:n], e[:n]))
        else:
            nb = oracle.Band.__new__(oracle.Band)
            nb.t, nb.f, nb.var, nb.uf = [np.zeros(0) for _ in range(4)]
            nb.up = np.zeros(0, np.uint8)
            bands.append(nb)
    rng = np.random.default_rng(100 * m + particles)
    lo, hi = [np.array(v) for v in BOUNDS[m]]
    P = rng.uniform(lo, hi, (len(bands), particles, lo.size))
    cat = lambda name, dt: torch.tensor(np.concatenate([getattr(b, name) for b in bands]).astype(dt), device="cuda")
    offs = torch.tensor(np.cumsum([0] + [b.n for b in bands]).astype(np.int32), device="cuda")
    dev = [cat("t", np.float64), cat("f", np.float64), cat("var", np.float64), cat("up", np.int32),
           cat("uf", np.float64), offs]
    pos = torch.tensor(P.reshape(-1), device="cuda")
    out = torch.full((len(bands) * particles,), float("nan"), dtype=torch.float64, device="cuda")
    L.launch_batch_pso_cost(*[x.data_ptr() for x in dev], pos.data_ptr(), out.data_ptr(), len(bands), particles,
                            lo.size, m, 1, 256)
    torch.cuda.synchronize()
    got = out.cpu().numpy().reshape(len(bands), particles)
    for i, b in enumerate(bands):
        ref = oracle.gpu_pso_cost(m, b, P[i]) if b.n else np.full(particles, 1e99)
        assert np.array_equal(got[i] >= 1e98, ref >= 1e98), i
        fin = ref < 1e98
        assert np.allclose(got[i][fin], ref[fin], rtol=1e-11, atol=1e-12), (i, np.abs(got[i] - ref).max())
