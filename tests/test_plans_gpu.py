"""Plans of the solve: rows per lane."""
from dataclasses import replace

import numpy as np
import pytest

from channel_rl_gb300 import cases as C
from tests.helpers import FIELD_RTOL, oracle_for, regions, rel

pytestmark = pytest.mark.gpu


# lane counts that leave the last lanes without rows: 4 lanes of 9 and 5 rows, 8 of 17
@pytest.mark.parametrize("shape", ((16, 9, 12), (12, 9, 16), (16, 17, 12), (8, 17, 8)))
def test_lanes_without_rows(shape):
    from channel_rl_gb300.host import Channel
    case = replace(C.smaller(C.c1_small(), *shape), LES_model=C.LES_NONE, amp=1.0)
    U, V, W = C.initial_fields(case)
    o = oracle_for(case)
    o.set_fields(U, V, W)
    o.compute_projection_step()
    reg = regions(o.g)
    out = []
    for mode in (0, 3):
        ch = Channel(case)
        ch.set_tile_shapes(608, 608, mode)
        ch.upload(U, V, W)
        ch.compute_projection_step()
        out.append(ch.download())
        ch.close()
    for f in "UVW":
        r = reg[f][0], slice(1, -1), reg[f][2]
        assert rel(out[0][f][r], getattr(o, f)[1:, 1:, 1:][r]) < FIELD_RTOL, f
        assert np.array_equal(out[0][f], out[1][f]), f
