"""GPU: the Hermite-basis SPME is as exact in any unit of length: every output
relative to its own size, against the numpy restatement (oracle/hspme.py)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("unit", [1e-4, 1.0, 1e4])
@pytest.mark.parametrize("box", [(7.0, 8.5, 6.2), (6.0, 6.0, 24.0)])
def test_outputs_in_other_units(mdf, unit, box):
    import torch
    from oracle.hspme import HermiteSPME as Orc
    rng = np.random.default_rng(3)
    n, K, CC, nbin = 40, (16, 15, 36 if box[2] > 20 else 18), 2.0, 8
    L = np.array(box) * unit
    x, q = rng.uniform(0, 1, (n, 3)), rng.choice([-1.0, 1.0], n)
    c = mdf.optibasis.bspline_initial_basis(CC, nbin, 4)
    dev = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
    hs = mdf.optibasis.HermiteSPME(n, K, L, 1.1 / unit, CC, nbin)
    out = hs.energy(dev(q), dev(x * L), dev(c[None]), forces=True, grads=True)
    E, F, dq, dr, dc = Orc(K, L, 1.1 / unit, CC, nbin, False).energy_grad(c, q, x * L)
    got = {k: v[0].cpu().numpy() for k, v in out.items()}
    # sums of at most 64 stencil points of transforms of 10^4 points, with stencil
    # coordinates K frac(x / L) rounded to 36 units of 1.1e-16: some 1e-14 of the largest value
    tol = 5e-14
    assert abs(got["energy"] - E) <= tol * abs(E)
    for d in range(3):
        assert np.abs(got["forces"][:, d] - F[:, d]).max() <= tol * np.abs(F[:, d]).max(), d
    for key, w in (("dE_dq", dq), ("dE_dr", dr), ("dE_dc", dc)):
        assert np.abs(got[key] - w).max() <= tol * np.abs(w).max(), key
