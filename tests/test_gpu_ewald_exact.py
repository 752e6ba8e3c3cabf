"""GPU: the exact reciprocal Ewald sum at the edges of its tiles (atoms and mode
rows around the staged sizes, odd and empty mode boxes, both precisions)
against the plain sum over modes in numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def plain(pos, q, box, K, beta):
    M = [k // 2 for k in K]
    m = np.stack(np.meshgrid(*[np.arange(-a, a + 1) for a in M], indexing="ij"), -1).reshape(-1, 3)
    m = m[(m != 0).any(1)] / box
    V, F, E = box.prod(), np.zeros_like(pos), 0.0
    for c in np.array_split(m, max(1, len(m) // 4096)):
        if not len(c):
            continue
        ph = 2 * np.pi * (c @ pos.T)
        cs, sn = np.cos(ph), np.sin(ph)
        mm = (c ** 2).sum(1)
        ex = np.exp(-(np.pi / beta) ** 2 * mm) / mm
        sr, si = cs @ q, sn @ q
        E += (ex * (sr ** 2 + si ** 2)).sum() / (2 * np.pi * V)
        F += q[:, None] * (((2 / V * ex)[:, None] * (sr[:, None] * sn - si[:, None] * cs)).T @ c)
    return E, F


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n,K", [(1, (8, 8, 8)), (31, (1, 1, 1)), (33, (2, 31, 5)), (129, (7, 6, 33)),
                                 (300, (16, 15, 14)), (257, (4, 3, 130))])
def test_ewald_exact_edges(mdf, n, K, prec):
    rng = np.random.default_rng(n)
    box = np.array([9.0, 7.5, 12.0])
    pos = (rng.uniform(0, 1, (n, 3)) * box).astype(np.float32).astype(np.float64)
    q = rng.choice([-1.0, 0.0, 1.0, 2.0], n)
    sys = mdf.MDSystem(pos, box, charge=q, precision=prec)
    mdf.InteractionEngine(sys).clearInteraction()
    E = mdf.ewald_exact(sys, K, 1.1)
    Eo, Fo = plain(pos, q, box, K, 1.1)
    # phases are reduced exactly: rounding of some 1e3 terms of binary64
    assert abs(E - Eo) <= 1e-12 * max(abs(Eo), 1e-3)
    assert np.abs(sys.forces() - Fo).max() <= 1e-12 * max(np.abs(Fo).max(), 1e-3)
    assert mdf.ewald_exact(sys, K, 1.1, add_forces=False) == E


def test_ewald_exact_many_atoms(mdf):
    """more atoms than one pass of the tables holds"""
    rng = np.random.default_rng(1)
    n, box = 65536 + 77, np.array([30.0, 31.0, 32.0])
    pos = rng.uniform(0, 1, (n, 3)) * box
    q = rng.choice([-1.0, 1.0], n)
    sys = mdf.MDSystem(pos, box, charge=q, precision=1)
    mdf.InteractionEngine(sys).clearInteraction()
    E = mdf.ewald_exact(sys, (3, 4, 2), 1.1)
    Eo, Fo = plain(pos, q, box, (3, 4, 2), 1.1)
    assert abs(E - Eo) <= 1e-10 * abs(Eo)
    assert np.abs(sys.forces() - Fo).max() <= 1e-10 * np.abs(Fo).max()


def test_ewald_exact_refuses_negative(mdf):
    sys = mdf.MDSystem(np.zeros((1, 3)), np.ones(3) * 5.0, charge=np.ones(1), precision=1)
    with pytest.raises(ValueError):
        mdf.ewald_exact(sys, (-4, 4, 4), 1.0)
