"""Zeros through the fixed-point kernels: what FP64 leaves exactly zero stays zero."""
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
