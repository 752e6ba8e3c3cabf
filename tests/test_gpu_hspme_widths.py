"""GPU: the batched Hermite-basis SPME at every stencil width, odd meshes and
candidate counts around a batch, with remainders of the atoms per warp,
against the numpy restatement (oracle/hspme.py)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,K,CC,nbin,C,bound0", [(1, (8, 8, 8), 1.0, 4, 1, False), (5, (9, 8, 7), 2.0, 3, 2, True),
                                                  (17, (8, 10, 12), 2.5, 5, 3, False), (9, (16, 8, 9), 3.0, 4, 5, False),
                                                  (6, (9, 12, 16), 4.0, 6, 4, True), (5, (11, 12, 13), 5.0, 4, 2, False),
                                                  (3, (16, 13, 14), 6.0, 5, 1, False), (3, (16, 15, 17), 7.0, 7, 3, False),
                                                  (2, (17, 18, 32), 8.0, 8, 2, True)])
def test_widths_and_batches(mdf, n, K, CC, nbin, C, bound0):
    import torch
    from oracle.hspme import HermiteSPME as Orc
    rng = np.random.default_rng(n + nbin)
    L = np.array([7.0, 8.5, 6.2])
    pos, q = rng.uniform(-1, 9, (n, 3)), rng.choice([-1.0, 1.0, 0.5], n)
    fref = rng.normal(0, 0.2, (n, 3))
    order = int(2 * np.ceil(CC))
    base = mdf.optibasis.bspline_initial_basis(CC, nbin, order, bound0=bound0)
    c = np.tile(base, (C, 1)) * (1 + 0.05 * rng.normal(size=(C, base.size)))
    dev = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
    hs = mdf.optibasis.HermiteSPME(n, K, L, 1.1, CC, nbin, bound0=bound0)
    a = hs.energy(dev(q), dev(pos), dev(c), forces=True, grads=True)
    b = hs.force_error(dev(q), dev(pos), dev(c), dev(fref))
    e_only = hs.energy(dev(q), dev(pos), dev(c))["energy"].cpu().numpy()
    o = Orc(K, L, 1.1, CC, nbin, bound0)
    for k in range(C):
        E, F, dq, dr, dc = o.energy_grad(c[k], q, pos)
        Lo, lq, lr, lc = o.force_error_grad(c[k], q, pos, fref)
        want = {"energy": E, "forces": F, "dE_dq": dq, "dE_dr": dr, "dE_dc": dc}
        for key, w in want.items():
            got = a[key][k].cpu().numpy()
            assert np.abs(got - w).max() <= 1e-11 * max(np.abs(w).max(), np.abs(F).max(), abs(E)), (key, k)
        for key, w in {"loss": Lo, "dL_dq": lq, "dL_dr": lr, "dL_dc": lc}.items():
            got = b[key][k].cpu().numpy()
            assert np.abs(got - w).max() <= 1e-11 * max(np.abs(w).max(), abs(Lo)), (key, k)
        assert abs(e_only[k] - E) <= 1e-12 * abs(E)
