"""GPU: the FP64 grid transforms under the error map, at every class of axis
length (powers of two, primes, composite lengths by their smallest factor,
lengths that change the lines per block), against the oracle's map."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [(2, 3, 4), (9, 16, 22), (13, 8, 49), (4, 97, 5), (2, 3, 121), (161, 2, 3), (3, 169, 2),
                               (205, 3, 2), (2, 2, 397), (1023, 2, 3), (2, 1024, 2), (64, 32, 128)])
def test_error_map_axis_lengths(mdf, orc, K):
    rng = np.random.default_rng(sum(K))
    box = tuple(0.4 * k for k in K)
    rho1, rho2 = rng.normal(0, 5, K), np.abs(rng.normal(30, 5, K))
    em = mdf.ErrorEstimate_SPME_Ik(K, box, 2.0, 4)
    em.set_profile(rho1, rho2)
    e1, e2 = em.calError(1.2)
    o1, o2 = orc.spme_ik_errmap(K, box, 2.0, 4, rho1, rho2, 1.2)
    for a, b in ((e1, o1), (e2, o2)):
        scale = np.abs(b[..., 0]).max()
        assert np.abs(a[..., 0] - b[..., 0]).max() < 1e-11 * scale
        assert np.abs(a[..., 1] - b[..., 1]).max() < 1e-9 * scale
    with np.errstate(invalid="ignore"):
        want = np.sqrt(e1[..., 0] + e2[..., 0])
    np.testing.assert_allclose(em.rms(1.2), want, rtol=1e-14, atol=0)


def test_maps_made_and_dropped_in_a_loop(mdf):
    """handles share the device's pool: a second map beside the first keeps its own values"""
    rng = np.random.default_rng(0)
    K, box = (16, 16, 16), (5.0, 5.0, 5.0)
    rho = rng.normal(0, 5, K), np.abs(rng.normal(30, 5, K))
    first = mdf.ErrorEstimate_SPME_Ik(K, box, 2.0, 4)
    first.set_profile(*rho)
    want = first.rms(1.0)
    for beta in (1.0, 1.5, 2.0):
        em = mdf.ErrorEstimate_SPME_Ik(K, box, beta, 4)
        em.set_profile(*rho)
        last = em.rms(1.0)
        del em
    np.testing.assert_array_equal(last, want)
    np.testing.assert_array_equal(first.rms(1.0), want)
