"""The persistent decode kernel at widths that are no multiples of its 256-wide sweeps, against the oracle."""
import numpy as np
import pytest

import ferrum_cpu_b200 as fcb
from ferrum_cpu_b200 import synth
from tests import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,heads,ff", [(320, 5, 288), (640, 10, 2560), (448, 7, 1312)])
def test_feeds_take_whole_rows(d, heads, ff):
    sm = synth.SynthModel(2, d, heads, ff, 48, 515, seed=d, perturb=True)
    om, gm = O.OracleModel(sm), fcb.CudaSlm(sm.config, sm.weights)
    gm.set_decode_mode(0)
    ids = synth.token_ids(4, 5, 515)
    for n in (1, 5):
        assert np.abs(gm.prime(ids[:n]) - om.prime(ids[:n])).max() < 2e-5
    assert np.abs(gm.feed(7) - om.feed(7)).max() < 2e-5
    gm.close()
    om.close()
