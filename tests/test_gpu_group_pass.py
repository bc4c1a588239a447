"""Passes by groups of lanes (small lattices): the same chain as the oracle's and as
the pass with one thread per site or link, which a batch takes when its other chains
make the launch large."""
import numpy as np
import pytest

from klft_b200 import Batch, GaugeField

pytestmark = pytest.mark.gpu

BETA = {1: 1.0, 2: 2.3, 3: 5.7}
DELTA = {1: 0.1, 2: 0.3, 3: 0.1}


# sites per pass: a single one, ragged CTAs, and one lattice for every width of a
# group (32, 16, 8 lanes in FP64); hits: none, one, more than a window of the stream
# holds
@pytest.mark.parametrize("nc,L,nhits", [(1, [2, 2], 3), (1, [6, 4], 1), (1, [4, 6, 10], 70), (1, [14, 16, 16, 8], 2),
                                        (1, [14, 16, 16, 16], 45),
                                        (2, [2, 2, 2], 5), (2, [4, 6, 8], 47), (2, [4, 4, 4, 6], 0),
                                        (2, [14, 16, 16, 16], 45), (3, [2, 4], 9), (3, [8, 6, 10, 4], 33),
                                        (3, [12, 12, 12, 16], 11)])
def test_group_pass_follows_oracle(oracle, nc, L, nhits):
    from oracle.oracle import Lat
    lat = Lat(nc, L)
    U = oracle.init(lat, True, 77)
    g = GaugeField(L, nc, "fp64", "hot", 77)
    g.set_stream(19, 3)
    acc = g.metropolis(BETA[nc], DELTA[nc], nhits, 2)
    acc_o = oracle.metropolis(lat, U, BETA[nc], DELTA[nc], nhits, 2, 19, chain=3)
    np.testing.assert_array_equal(acc, np.nan_to_num(acc_o))  # no hits: the oracle's 0 / 0 is 0 here
    np.testing.assert_allclose(g.download(), U, rtol=0, atol=1e-11)


@pytest.mark.parametrize("nc", [1, 2, 3])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("L,defect", [([8, 6, 4, 10], 0), ([8, 6, 4, 10], 2), ([16, 16, 16, 26], 0), ([12, 10, 6], 0),
                                      ([20, 14], 0)])
def test_group_pass_is_the_chain_of_the_site_pass(nc, precision, L, defect):
    big = [24, 24, 24, 32] if len(L) == 4 else ([64, 56, 56] if len(L) == 3 else [320, 320])

    def field(ext, seed):
        g = GaugeField(ext, nc, precision, "hot", seed)
        g.set_stream(seed, 1)
        if defect:
            g.set_defect(defect, (0, 1, 0), 0.5)
        return g

    alone, member, other = field(L, 5), field(L, 5), field(big, 6)
    b = Batch()
    for g in (member, other):
        b.add(g, BETA[nc], DELTA[nc], 10)
    acc, _, _, _ = b.run(3, False, False)
    np.testing.assert_array_equal(alone.metropolis(BETA[nc], DELTA[nc], 10, 3), acc[:, 0])
    np.testing.assert_array_equal(alone.download(), member.download())
    b.close()


# 16 lanes, 4 lanes, 3 and 2 dimensions; hits: fewer and more than the lanes
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("L,defect,nhits", [([8, 6, 4, 10], 0, 10), ([8, 6, 4, 10], 2, 37), ([8, 8, 8, 16], 0, 10),
                                            ([8, 8, 8, 16], 2, 6), ([10, 12, 14], 0, 37), ([20, 14], 0, 1)])
def test_exp_group_pass_is_the_chain_of_the_link_pass(precision, L, defect, nhits):
    big = [16, 16, 16, 8] if len(L) == 4 else ([32, 32, 16] if len(L) == 3 else [128, 128])

    def field(ext, seed):
        g = GaugeField(ext, 3, precision, "hot", seed)
        g.set_stream(seed, 1)
        if defect:
            g.set_defect(defect, (0, 1, 0), 0.5)
        return g

    alone, member, other = field(L, 5), field(L, 5), field(big, 6)
    b = Batch()
    for g in (member, other):
        b.add(g, 5.7, 0.0, nhits, "exp", 0.25)
    acc, _, _, _ = b.run(3, False, False)
    np.testing.assert_array_equal(alone.metropolis(5.7, 0.0, nhits, 3, "exp", 0.25), acc[:, 0])
    np.testing.assert_array_equal(alone.download(), member.download())
    b.close()


# FP32 U(1) and SU(2), where each lane runs the site's hits on links that lane 0 stores:
# one site to several CTAs, 4 and 8 lanes, hits that need no window, one, and several
# (so that a link's hits are resumed in a new window), and extents that leave the lanes
# of a group with different shares of the neighbours
@pytest.mark.parametrize("nc", [1, 2])
@pytest.mark.parametrize("L,nhits", [([2, 2], 47), ([6, 4], 11), ([4, 6, 10], 0), ([4, 6, 10], 47), ([2, 2, 2], 30),
                                     ([6, 2, 4, 2], 1), ([4, 4, 4, 6], 11), ([8, 6, 4, 10], 47), ([40, 44, 48], 11)])
def test_fp32_group_pass_resumes_hits_and_orders_stores(nc, L, nhits):
    big = {4: [24, 24, 24, 32], 3: [64, 56, 56], 2: [320, 320]}[len(L)]
    fields = []
    for ext, seed in ((L, 5), (L, 5), (big, 6)):
        g = GaugeField(ext, nc, "mixed", "hot", seed)
        g.set_stream(seed, 1)
        fields.append(g)
    alone, member, other = fields
    b = Batch()
    for g in (member, other):
        b.add(g, BETA[nc], DELTA[nc], nhits)
    acc, _, _, _ = b.run(4, False, False)
    np.testing.assert_array_equal(alone.metropolis(BETA[nc], DELTA[nc], nhits, 4), acc[:, 0])
    np.testing.assert_array_equal(alone.download(), member.download())
    b.close()


# SU(3) in FP32 where many hits are accepted (strong coupling, disordered links) and 10^8 are
# drawn: a staple whose last bit differs changes one decision in 10^7
@pytest.mark.parametrize("L,defect,beta", [([16, 16, 12, 12], 0, 0.5), ([16, 16, 12, 12], 0, 2.0),
                                           ([16, 16, 12, 12], 2, 2.0), ([24, 20, 36], 0, 1.0)])
def test_su3_fp32_group_pass_at_strong_coupling(L, defect, beta):
    big = [24, 24, 24, 32] if len(L) == 4 else [64, 56, 56]
    fields = []
    for ext, seed in ((L, 5), (L, 5), (big, 6)):
        g = GaugeField(ext, 3, "mixed", "hot", seed)
        g.set_stream(seed, 1)
        if defect:
            g.set_defect(defect, (0, 1, 0), 0.5)
        fields.append(g)
    alone, member, other = fields
    b = Batch()
    for g in (member, other):
        b.add(g, beta, 0.1, 40)
    acc, _, _, _ = b.run(20, False, False)
    np.testing.assert_array_equal(alone.metropolis(beta, 0.1, 40, 20), acc[:, 0])
    np.testing.assert_array_equal(alone.download(), member.download())
    b.close()
