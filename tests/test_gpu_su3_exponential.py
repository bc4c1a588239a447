"""exp(iQ) of SU(3) where its argument is halved more than once (c1 = Tr Q^2 / 2 above 3): large
proposal widths and molecular-dynamics steps."""
import numpy as np
import pytest

from klft_b200 import GaugeField
from oracle.oracle import Lat

pytestmark = pytest.mark.gpu

# c1 averages 2 eps^2: 2, 8 and 32, that is one to six halvings
EPS = [1.0, 2.0, 4.0]


def off_unitary(u):
    return np.abs(u @ u.conj().swapaxes(-1, -2) - np.eye(3)).max()


@pytest.mark.parametrize("eps", EPS)
@pytest.mark.parametrize("L", [[4, 6], [4, 4, 6], [4, 2, 6, 4], [16, 16, 14]])
def test_wide_exp_proposals_match_oracle(oracle, L, eps):
    lat = Lat(3, L)
    U = oracle.init(lat, True, 71)
    g = GaugeField(L, 3, "fp64", "hot", 71)
    g.set_stream(7, 2)
    acc = g.metropolis(3.0, 0.0, 5, 3, "exp", eps)
    acc_o = oracle.metropolis(lat, U, 3.0, 0.0, 5, 3, 7, chain=2, proposal=1, eps=eps)
    np.testing.assert_array_equal(acc, acc_o)
    np.testing.assert_allclose(g.download(), U, rtol=0, atol=1e-11)


# one thread per link and groups of lanes; FP32 links are stored as two rows, normalised to FP32
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-13), ("mixed", 5e-6)])
@pytest.mark.parametrize("eps", EPS)
@pytest.mark.parametrize("L", [[8, 6, 4, 10], [16, 16, 16, 12]])
def test_wide_exp_proposals_stay_in_the_group(L, eps, precision, tol):
    g = GaugeField(L, 3, precision, "hot", 72)
    g.metropolis(3.0, 0.0, 10, 6, "exp", eps)
    assert off_unitary(g.download()) < tol


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 2e-5)])
@pytest.mark.parametrize("tau", [0.5, 1.5, 4.0])
def test_long_link_updates_match_oracle(oracle, tau, precision, tol):
    """beta = 0: the momenta stay, one leapfrog step multiplies each link by exp(i tau p)."""
    L = [6, 4, 4, 2]
    lat = Lat(3, L)
    U = oracle.init(lat, True, 73)
    P = np.random.default_rng(9).normal(size=(lat.V, 4, 8))
    g = GaugeField(L, 3, precision, "cold", 1)
    g.upload(U)
    g.set_momenta(P)
    g.hmc_integrate(0.0, tau, 1, "leapfrog")
    oracle.integrate(lat, U, P, 0.0, tau, 1, 1)
    np.testing.assert_allclose(g.download(), U, rtol=0, atol=tol)
