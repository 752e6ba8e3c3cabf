"""GPU: the particle-mesh kernels at the edges of their tiles and lane
mappings -- charges per warp and atoms per gather group with remainders,
neutral atoms, clustered and scattered charges (tile and direct paths), every
class of order -- against the CPU oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOX = np.array([9.0, 9.0, 9.0])


def rel(a, b):
    return float(np.sqrt(((a - b) ** 2).sum() / (b ** 2).sum()))


def cloud(n, spread, seed):
    """n charges around a corner of the box (periodic images in one warp) or all over it"""
    rng = np.random.default_rng(seed)
    pos = np.mod(rng.normal(0.0, spread, (n, 3)), BOX) if spread else rng.uniform(0, BOX, (n, 3))
    pos = pos.astype(np.float32).astype(np.float64)
    pos[pos >= BOX] = 0.0
    q = rng.choice([-1.0, 0.0, 1.0, 2.0], n)
    q[0] = 1.0
    return pos, q


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n,spread,order,K", [(1, 0.3, 6, (16, 16, 32)), (15, 0.3, 6, (16, 16, 32)),
                                              (33, 0.0, 6, (32, 16, 16)), (200, 0.4, 6, (64, 64, 64)),
                                              (67, 0.5, 2, (8, 8, 8)), (65, 0.5, 3, (8, 16, 4)), (70, 0.5, 4, (16, 8, 8)),
                                              (66, 0.5, 5, (16, 16, 16)), (71, 0.5, 7, (8, 8, 16)),
                                              (64, 0.5, 8, (16, 16, 16)), (40, 0.5, 9, (16, 32, 16)),
                                              (40, 0.5, 12, (16, 16, 16)), (40, 0.0, 14, (16, 16, 32))])
def test_mesh_and_forces(mdf, orc, n, spread, order, K, prec):
    pos, q = cloud(n, spread, n + order)
    sys = mdf.MDSystem(pos, BOX, charge=q, precision=prec)
    eng = mdf.InteractionEngine(sys)
    for method, code in (("ik", 0), ("analytic", 1)):
        sp = mdf.SPME(sys, K, order, 1.2, method)
        Qo = orc.spme_spread(pos, q, BOX, K, order)
        # binary32: order^3 products of three rounded weights per charge
        assert np.abs(sp.mesh() - Qo).max() < (2e-5 if prec == 0 else 1e-12)
        if order % 2:
            continue  # |b(m)|^2 is infinite at the Nyquist index of an odd order: no forces to compare
        eng.clearInteraction()
        sp.apply()
        _, Fo = orc.spme_rec(pos, q, BOX, K, order, 1.2, code)
        F = sys.forces()
        # order 8 and above: the oracle's recursion and the reference's tables agree to 1e-9
        assert np.sqrt(((F - Fo) ** 2).sum()) <= (2e-5 if prec == 0 else 1e-9) * max(np.sqrt((Fo ** 2).sum()), 0.1)
        assert (F[q == 0] == 0).all()
        # the adjoint's exact gradient is minus the analytic force
        if method == "analytic":
            g = sp.energy_grad()
            assert np.sqrt(((g["dE_dr"] + Fo) ** 2).sum()) <= (2e-5 if prec == 0 else 1e-9) * max(
                np.sqrt((Fo ** 2).sum()), 0.1)
            assert abs(0.5 * (q * g["dE_dq"]).sum() - g["energy"]) <= (2e-5 if prec == 0 else 1e-11) * abs(g["energy"])


@pytest.mark.parametrize("n,order,prec", [(200000, 6, 0), (200017, 5, 0), (220000, 4, 0), (200000, 6, 1)])
@pytest.mark.parametrize("sort", [True, False])
def test_large_dense_spread(mdf, orc, n, order, prec, sort):
    """the tiles of the large dense systems, in cell order and scattered (no tile fits)"""
    rng = np.random.default_rng(n)
    box = np.array([60.0, 60.0, 60.0])
    pos = rng.uniform(0, 60.0, (n, 3)).astype(np.float32).astype(np.float64)
    pos[pos >= 60.0] = 0.0
    q = rng.choice([-1.0, 0.0, 1.0], n)
    sys = mdf.MDSystem(pos, box, charge=q, precision=prec)
    if sort:
        cl = mdf.CellList(sys, 2.8)
        cl.rebuild()
    K = (64, 128, 128)
    sp = mdf.SPME(sys, K, order, 1.0)
    assert np.abs(sp.mesh() - orc.spme_spread(pos, q, box, K, order)).max() < (2e-5 if prec == 0 else 1e-12)
