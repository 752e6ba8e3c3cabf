"""GPU: SPME gradients and virials on the larger planes, the spread's tile at high
orders, energies without gradients, and gradients on two streams in turn."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {0: 2e-5, 1: 1e-10}


def charges(n, box, seed):
    rng = np.random.default_rng(seed)
    pos = (rng.uniform(0, 1, (n, 3)) * box).astype(np.float32).astype(np.float64)
    pos[pos >= box] = 0.0
    return pos, rng.choice([-1.0, 1.0, 0.0], n)


@pytest.fixture(scope="module")
def oracle(orc):
    """energy and forces by case: the oracle's transforms take seconds, and both precisions ask for the same"""
    kept = {}

    def rec(pos, q, box, K, order, method, scale=0.0):
        key = (len(pos), K, order, method, scale)
        if key not in kept:
            kept[key] = orc.spme_rec(pos * (1 + scale), q, box * (1 + scale), K, order, 1.1, method)
        return kept[key]

    return rec


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n,K,order", [(150, (64, 64, 128), 4), (4400, (128, 128, 64), 4), (2000, (64, 64, 256), 6),
                                       (4400, (64, 64, 256), 6), (150, (64, 32, 64), 4)])
def test_gradients_and_virial(mdf, oracle, n, K, order, prec):
    box = np.array([9.0, 8.0, 11.0])
    pos, q = charges(n, box, n + K[2])
    sys = mdf.MDSystem(pos, box, charge=q, precision=prec)
    sp = mdf.SPME(sys, K, order, 1.1)
    sys.clear_stats()
    sp.apply()
    st = sys.stats()
    Eo, _ = oracle(pos, q, box, K, order, 0)
    _, Fa = oracle(pos, q, box, K, order, 1)
    s = 1e-4
    Ep, Em = (oracle(pos, q, box, K, order, 0, x)[0] for x in (s, -s))
    w = st[[mdf.STAT_VIRIAL_XX, mdf.STAT_VIRIAL_YY, mdf.STAT_VIRIAL_ZZ]].sum()
    assert abs(w - (Ep - Em) / (2 * s)) <= (1e-4 if prec == 0 else 1e-6) * max(abs(w), abs(Eo))
    if K[0] * K[1] * (K[2] // 2 + 1) > 256 * (n // 4 + 1024):  # more mesh blocks than the gradient takes for n atoms
        with pytest.raises(mdf.core.MDExcptBadArgument):
            sp.energy_grad()
        return
    g, h = sp.energy_grad(), sp.energy_grad(dpsi=True)  # with dE/dpsi: the passes per axis
    assert abs(g["energy"] - Eo) <= TOL[prec] * abs(Eo)
    assert np.sqrt(((g["dE_dr"] + Fa) ** 2).sum()) <= TOL[prec] * np.sqrt((Fa ** 2).sum())
    for k in ("energy", "dE_dbeta", "dE_dq", "dE_dr"):
        np.testing.assert_allclose(g[k], h[k], rtol=0, atol=TOL[prec] * np.abs(h[k]).max())
    alone = sp.energy_grad(dq=False, dr=False)
    assert alone["energy"] == pytest.approx(g["energy"], rel=TOL[prec])
    assert alone["dE_dbeta"] == pytest.approx(g["dE_dbeta"], rel=10 * TOL[prec])
    again = sp.energy_grad()  # on the mesh that the energy alone cleared
    for k in ("dE_dq", "dE_dr"):
        np.testing.assert_allclose(again[k], g[k], rtol=0, atol=TOL[prec] * np.abs(g[k]).max())


@pytest.mark.parametrize("order", [8, 9, 11, 14])
@pytest.mark.parametrize("sort", [True, False])
def test_large_dense_spread_at_high_orders(mdf, orc, order, sort):
    """the tile with its rows in several rounds, and stencils that no tile holds"""
    n, box, K = 200003, np.array([40.0, 40.0, 40.0]), (64, 64, 64)
    pos, q = charges(n, box, order)
    sys = mdf.MDSystem(pos, box, charge=q, precision=0)
    if sort:
        cl = mdf.CellList(sys, 2.8)
        cl.rebuild()
    sp = mdf.SPME(sys, K, order, 1.0)
    Q = orc.spme_spread(pos, q, box, K, order)
    # some n order^3 / K^3 rounded products a point
    assert np.abs(sp.mesh() - Q).max() < 2e-5 * max(1.0, np.sqrt(n * order ** 3 / np.prod(K)) / 10)


def test_two_streams_in_turn(mdf):
    """the system follows torch's current stream; results on either are the same"""
    import torch
    box = np.array([9.0, 8.0, 11.0])
    pos, q = charges(900, box, 4)
    sys = mdf.MDSystem(pos, box, charge=q, precision=1)
    sp = mdf.SPME(sys, (32, 32, 64), 6, 1.1)
    streams = [torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.default_stream()]
    data = [(torch.tensor(q * (1 + 0.1 * k), device="cuda"), torch.tensor(pos, device="cuda")) for k in range(3)]
    torch.cuda.synchronize()

    def evaluate(k, stream):
        with torch.cuda.stream(stream):
            qt, rt = (t.clone().requires_grad_(True) for t in data[k])
            e = mdf.optibasis.spme_energy(qt, rt, sp, recompute=bool(k % 2))
            e.backward()
        return e.detach(), qt.grad, rt.grad

    want = []
    for k in range(3):
        want.append([t.cpu().numpy() for t in evaluate(k, streams[2])])
    for turn in range(12):
        k, stream = turn % 3, streams[(turn // 2) % 3]
        got = evaluate(k, stream)
        stream.synchronize()
        for g, w in zip(got, want[k]):
            np.testing.assert_allclose(g.cpu().numpy(), w, rtol=0, atol=1e-12 * np.abs(w).max())
