"""GPU: the SPME transforms by planes (equal x and y sizes) at every plane size
and z length, beside meshes that keep the passes per axis, against the CPU
oracle: energies, forces of both differentiation methods, virial, adjoint."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {0: 2e-5, 1: 1e-10}


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("K,order", [((16, 16, 4), 2), ((16, 16, 8), 4), ((16, 16, 16), 6), ((16, 16, 1024), 4),
                                     ((32, 32, 8), 4), ((32, 32, 256), 6), ((64, 64, 16), 6), ((64, 64, 128), 4),
                                     ((128, 128, 16), 6), ((128, 128, 64), 4), ((16, 16, 512), 6), ((8, 8, 16), 4),
                                     ((32, 16, 16), 6), ((16, 64, 32), 4)])
def test_planes_match_oracle(mdf, orc, K, order, prec):
    rng = np.random.default_rng(sum(K) + order)
    n, box = 150, np.array([9.0, 8.0, 11.0])
    pos = (rng.uniform(0, 1, (n, 3)) * box).astype(np.float32).astype(np.float64)
    q = rng.choice([-1.0, 1.0, 0.0], n)
    sys = mdf.MDSystem(pos, box, charge=q, precision=prec)
    eng = mdf.InteractionEngine(sys)
    for method, code in (("ik", 0), ("analytic", 1)):
        sp = mdf.SPME(sys, K, order, 1.1, method)
        for _ in range(2):  # the second pass on the mesh the first one cleared
            eng.clearInteraction()
            sys.clear_stats()
            sp.apply()
        Eo, Fo = orc.spme_rec(pos, q, box, K, order, 1.1, code)
        F, st = sys.forces(), sys.stats()
        assert abs(st[mdf.STAT_ELEC_REC] - Eo) <= TOL[prec] * abs(Eo)
        assert np.sqrt(((F - Fo) ** 2).sum()) <= TOL[prec] * np.sqrt((Fo ** 2).sum())
        eng.clearInteraction()
        sp.apply(with_stats=False)
        np.testing.assert_allclose(sys.forces(), F, rtol=0, atol=TOL[prec] * np.abs(F).max())
    if K[0] * K[1] * (K[2] // 2 + 1) > 256 * 1024:
        return  # more mesh blocks than the gradient takes for a system of this size (refused)
    g, h = sp.energy_grad(), sp.energy_grad(dpsi=True)  # with dE/dpsi: the passes per axis
    assert abs(g["energy"] - Eo) <= TOL[prec] * abs(Eo)
    assert np.sqrt(((g["dE_dr"] + Fo) ** 2).sum()) <= TOL[prec] * np.sqrt((Fo ** 2).sum())
    for k in ("energy", "dE_dbeta", "dE_dq", "dE_dr"):
        np.testing.assert_allclose(g[k], h[k], rtol=0, atol=TOL[prec] * np.abs(h[k]).max())
    # the virial is the energy's response to a scaled box, V P = -dE/ds at fixed charges
    s = 1e-4
    Ep = orc.spme_rec(pos * (1 + s), q, box * (1 + s), K, order, 1.1, 0)[0]
    Em = orc.spme_rec(pos * (1 - s), q, box * (1 - s), K, order, 1.1, 0)[0]
    w = st[[mdf.STAT_VIRIAL_XX, mdf.STAT_VIRIAL_YY, mdf.STAT_VIRIAL_ZZ]].sum()
    assert abs(w - (Ep - Em) / (2 * s)) <= (1e-4 if prec == 0 else 1e-6) * max(abs(w), abs(Eo))
