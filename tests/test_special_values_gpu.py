"""Zeros, tiny and huge velocities through the fixed-point kernels: what FP64
leaves exactly zero stays zero, what overflows there is flagged."""
from dataclasses import replace

import numpy as np
import pytest

from channel_rl_gb300 import cases as C

pytestmark = pytest.mark.gpu


def test_zeros_of_either_sign_project_to_zero():
    """The differences of zeros are zero, so no correction is made."""
    from channel_rl_gb300.host import Channel
    case = replace(C.smaller(C.c1_small(), 16, 9, 12), LES_model=C.LES_NONE, x_mass_cte=0)
    rng = np.random.default_rng(3)
    f = [np.copysign(0.0 * a, rng.random(a.shape) - 0.5) for a in C.initial_fields(case)]
    ch = Channel(case)
    ch.upload(*(np.asfortranarray(a) for a in f))
    ch.compute_projection_step()
    d, p = ch.download(), ch.pseudo_pressure()
    ch.close()
    assert all(not d[q].any() for q in "UVW") and not p.any()


@pytest.mark.parametrize("les,wm", ((C.LES_NONE, C.WM_NONE), (C.LES_SMAG, C.WM_NONE), (C.LES_DSM, C.WM_EQLOG), (C.LES_AMD, C.WM_NONE)))
def test_velocities_whose_products_overflow_are_flagged(les, wm):
    """On a grid with spacings above 1, where only the products U U exceed a
    double's range and no later factor does."""
    from channel_rl_gb300.host import Channel, ChlError
    base = C.wallmodelled("o", 16, 12, 16, 2000.0, les=les, wall_model=wm)
    x, y, z = (1e3 * a for a in C.faces(base))
    case = replace(base, xf=tuple(x), yf=tuple(y), zf=tuple(z), CFL=-1e-6)
    ch = Channel(case)
    ch.upload(*(1e160 * a for a in C.initial_fields(base)))
    ch.step(3)
    with pytest.raises(ChlError):
        ch.synchronize()
    ch.close()
