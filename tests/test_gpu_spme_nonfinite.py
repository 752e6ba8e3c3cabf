"""GPU: coordinates that are no numbers (a diverged optimisation) stay inside the
mesh kernels' memory: the energy is no number either, and the object works on."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("K", [(16, 16, 32), (32, 16, 16)])
def test_nonfinite_coordinates(mdf, bad, K, prec):
    import torch
    rng = np.random.default_rng(8)
    n, box = 70, np.array([9.0, 8.0, 11.0])
    pos = rng.uniform(0, 1, (n, 3)) * box
    q = rng.choice([-1.0, 1.0], n)
    sys = mdf.MDSystem(pos, box, charge=q, precision=prec)
    eng = mdf.InteractionEngine(sys)
    sp = mdf.SPME(sys, K, 6, 1.1)

    def evaluate(p):
        qt = torch.tensor(q, device="cuda", requires_grad=True)
        rt = torch.tensor(p, device="cuda", requires_grad=True)
        e = mdf.optibasis.spme_energy(qt, rt, sp)
        e.backward()
        eng.clearInteraction()
        sp.apply()
        return e.item(), rt.grad.cpu().numpy(), sys.forces()

    want = evaluate(pos)
    for i, d in ((33, 0), (0, 1), (n - 1, 2)):
        p = pos.copy()
        p[i, d] = bad
        assert np.isnan(evaluate(p)[0])
    got = evaluate(pos)
    for w, g in zip(want, got):
        np.testing.assert_allclose(g, w, rtol=0, atol=(2e-5 if prec == 0 else 1e-12) * np.abs(w).max())
