"""GPU: value and gradient of the optiBasis error functional where the
kernel can go wrong: odd and tiny meshes (the mirror pairs and the doubled
edges of an even axis), coefficient counts around the groups of four and 32
that are worked on together, candidate counts, one image and several; against
the oracle, in double precision (1e-10 of the value, 1e-10 of the largest
gradient component: a few thousand terms of like sign)."""
import numpy as np
import pytest

from oracle.ikerror import IkErrorOracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,nbin,bound0,l_cut,C", [((2, 3, 4), 2, False, 1, 1), ((5, 8, 13), 2, True, 2, 3),
                                                   ((16, 7, 9), 5, False, 3, 2), ((12, 12, 12), 17, True, 10, 9),
                                                   ((24, 15, 32), 21, False, 4, 4)])
def test_value_and_gradient(mdf, K, nbin, bound0, l_cut, C):
    CC, beta, L, q2, n = 3.0, 1.1, [0.9 * k for k in K], 50.0, 40.0
    cls = mdf.optibasis.HermiteLossFunc_Bound0 if bound0 else mdf.optibasis.HermiteLossFunc
    f = cls(CC, nbin, beta, list(K), q2, n, L, l_cut=l_cut)
    o = IkErrorOracle(CC, nbin, beta, list(K), L, q2, n, l_cut, bound0)
    rng = np.random.default_rng(nbin)
    base = mdf.optibasis.bspline_initial_basis(CC, nbin, 6, bound0=bound0)
    V = base[None, :] * (1 + 0.02 * rng.normal(size=(C, base.size)))
    val, g = f.evaluate(V)
    only = f.evaluate(V, grads=False)
    for c in range(C):
        want = o.value(V[c])
        assert abs(val[c] - want) < 1e-10 * want
        w = np.asarray(o.deriv(V[c]))
        assert np.abs(g[c] - w).max() < 1e-10 * np.abs(w).max()
    assert np.array_equal(only[0] if isinstance(only, tuple) else only, val)
