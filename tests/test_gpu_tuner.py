"""The launch-shape tuner and passes by groups of lanes, whose launch shape is fixed: their keys
are kept with it, and no candidate is timed (a timed one would be any of 32, 64 and 128)."""
import pytest

import klft_b200
from klft_b200._lib import lib

pytestmark = pytest.mark.gpu

BETA = {1: 1.0, 2: 2.3, 3: 5.7}


def test_group_passes_have_nothing_to_tune(tmp_path):
    cache = str(tmp_path / "tune.txt")
    kinds = [(nc, prec, "reference") for nc in (1, 2, 3) for prec in ("fp64", "mixed")]
    kinds += [(3, "fp64", "exp"), (3, "mixed", "exp")]
    extents = ([4, 4, 4, 4], [8, 8, 8, 8], [8, 6, 10], [16, 12])
    try:
        lib().klft_tuner_clear()
        lib().klft_tuner_configure(1, 0)
        for nc, prec, proposal in kinds:
            fields = []
            b = klft_b200.Batch()
            for k, L in enumerate(extents):
                g = klft_b200.GaugeField(L, nc, prec, "hot", 3 + k)
                g.metropolis(BETA[nc], 0.2, 4, 1, proposal, 0.2)
                b.add(g, BETA[nc], 0.2, 4, proposal, 0.2)
                fields.append(g)
            b.run(1)
            b.close()
        assert lib().klft_tuner_write_cache(cache.encode()) == 0
    finally:
        lib().klft_tuner_configure(0, 0)
        lib().klft_tuner_clear()
    got = [line.split() for line in open(cache)]
    assert len(got) == len(kinds) * (len(extents) + 1)
    assert {int(line[2]) for line in got} == {128}, got
