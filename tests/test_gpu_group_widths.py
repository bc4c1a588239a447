"""A pass by groups of lanes is taken only where it is the faster one: a lattice that the
rule gives to groups takes no longer than a larger one that has a thread per site, whose
pass is bound by one site's chain of hits.  Few and many hits, strong coupling."""
import time

import pytest

from klft_b200 import GaugeField

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc,precision,beta,delta,nhits,L,larger", [
    (3, "fp64", 0.5, 0.1, 10, [16, 16, 16, 32], [16, 16, 24, 32]),
    (3, "mixed", 0.5, 0.1, 10, [16, 16, 16, 32], [16, 16, 24, 32]),
    (2, "fp64", 2.3, 0.3, 1, [16, 16, 16, 16], [16, 16, 16, 26]),
    (1, "mixed", 2.0, 0.1, 30, [16, 16, 16, 36], [16, 16, 32, 34]),
])
def test_groups_of_lanes_where_they_are_faster(nc, precision, beta, delta, nhits, L, larger):
    def sweep_time(ext):
        g = GaugeField(ext, nc, precision, "hot", 3)
        g.metropolis(beta, delta, nhits, 10)
        best = 1e9
        for _ in range(5):
            t = time.perf_counter()
            g.metropolis(beta, delta, nhits, 10)
            best = min(best, time.perf_counter() - t)
        return best

    assert sweep_time(L) < 1.2 * sweep_time(larger)
