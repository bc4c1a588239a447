"""Axial gauge of U(1) and SU(2) temporal loops on both sides of the column count from which a
column is one thread's (80,000 and 48,000 columns), against the oracle."""
import numpy as np
import pytest

from klft_b200 import GaugeField
from oracle.oracle import Lat

pytestmark = pytest.mark.gpu

TOL = {"mixed": dict(rtol=0, atol=2e-6), "fp64": dict(rtol=1e-12, atol=1e-14)}


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("nc,L", [(1, [40, 44, 44, 4]), (1, [44, 44, 44, 4]), (2, [36, 36, 36, 4]), (2, [40, 36, 36, 6])])
def test_loops_of_many_columns_match_oracle(oracle, nc, L, precision):
    lat = Lat(nc, L)
    U = oracle.init(lat, True, 51)
    g = GaugeField(L, nc, precision)
    g.upload(U)
    pairs = [(1, 1), (2, 3), (3, 2)]
    np.testing.assert_allclose(g.wilson_loop_temporal(pairs), oracle.wilson_temporal(lat, U, pairs), **TOL[precision])
    g.close()
