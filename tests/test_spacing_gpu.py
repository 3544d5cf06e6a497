"""Grids that are uniform in x and z only to the accepted 1e-9: the strain takes
every edge's own spacing, as compute_Sij does."""
from dataclasses import replace

import numpy as np
import pytest

from channel_rl_gb300 import cases as C
from tests.helpers import FIELD_RTOL, NUT_RTOL, oracle_for, regions, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("les,shape,tol", ((C.LES_SMAG, (18, 9, 12), FIELD_RTOL), (C.LES_SMAG, (54, 12, 36), FIELD_RTOL),
                                           (C.LES_VREMAN, (18, 9, 12), NUT_RTOL), (C.LES_DSM, (16, 9, 12), NUT_RTOL)))
def test_edges_keep_their_own_spacing(les, shape, tol):
    """FIELD_RTOL for the static model; NUT_RTOL where B_b or the plane sums cancel."""
    from channel_rl_gb300.host import Channel
    case = replace(C.smaller(C.c1_small(), *shape), LES_model=les, x_mass_cte=0, dPdx=1e-3)
    x, y, z = C.faces(case)
    rng = np.random.default_rng(11)
    for f in (x, z):            # the faces around the periodic seam stay: the ghost centres mirror there
        f[2:-4] += 0.45e-9 * (f[1] - f[0]) * rng.choice((-1.0, 1.0), f.size - 6)
    U, V, W = C.initial_fields(case)
    case = replace(case, xf=tuple(x), yf=tuple(y), zf=tuple(z))
    o = oracle_for(case)
    o.set_fields(U, V, W)
    o.compute_eddy_viscosity()
    ch = Channel(case)
    ch.upload(U, V, W)
    ch.compute_eddy_viscosity()
    nt = ch.download(fields=("nu_t",))["nu_t"]
    ch.close()
    reg = regions(o.g)["C"]
    assert rel(nt[reg], o.nu_t[1:, 1:, 1:][reg]) < tol
