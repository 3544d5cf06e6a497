"""Eddy viscosities where the terms of a model differ by many orders of magnitude:
nearly parallel flows, and the rows next to resolved walls.  nu is tiny, because
nu_t is read back as the stored nu + nu_t less nu."""
from dataclasses import replace

import numpy as np
import pytest

from channel_rl_gb300 import cases as C
from tests.helpers import FIELD_RTOL, NUT_RTOL, oracle_for

pytestmark = pytest.mark.gpu


def _nu_t(case, U, V, W):
    from channel_rl_gb300.host import Channel
    o = oracle_for(case)
    o.set_fields(U, V, W)
    o.compute_eddy_viscosity()
    ch = Channel(case)
    ch.upload(U, V, W)
    ch.compute_eddy_viscosity()
    got = ch.download(fields=("nu_t",))["nu_t"]
    ch.close()
    cut = slice(1, case.Nx + 1), slice(1, case.Ny + 1), slice(1, case.Nz + 1)
    return got[cut], o.nu_t[1:, 1:, 1:][cut]


@pytest.mark.parametrize("amp", (1e-4, 1e-6, 1e-8))
@pytest.mark.parametrize("les", (C.LES_AMD, C.LES_VREMAN))
def test_nearly_parallel_flow(les, amp):
    """A laminar profile with noise of the given size: AMD's largest terms are the
    wall-normal gradient times the noise, Vreman's B_b is a product with it.
    FIELD_RTOL times the digits by which B_b cancels for Vreman (its b_11 b_22 and
    b_12^2 have the noise's own rounding in common)."""
    case = replace(C.smaller(C.c1_small(), 16, 12, 16), Lx=2.0, Lz=2.0, LES_model=les, x_mass_cte=0, dPdx=1e-3,
                   nu=1e-20, amp=amp, Dirichlet_nu_t=0)
    got, ref = _nu_t(case, *C.initial_fields(case))
    assert np.abs(got - ref).max() < FIELD_RTOL * np.abs(ref).max()


@pytest.mark.parametrize("shape,stretch", (((24, 24, 18), 2.5), ((16, 13, 12), 2.0)))
def test_dynamic_model_row_by_row_next_to_resolved_walls(shape, stretch):
    """U as the wall distance, V as its square: each row relative to its own."""
    case = replace(C.smaller(C.c1_small(), *shape), stretch=stretch, x_mass_cte=0, dPdx=1e-3, nu=1e-20,
                   Dirichlet_nu_t=0)
    U, V, W = (a.copy(order="F") for a in C.initial_fields(case))
    d, dg = (1.0 - np.abs(y) for y in (C.faces(case)[1], C.centres_y(C.faces(case)[1])))
    rng = np.random.default_rng(5)
    U *= 0
    U += (1.5 * dg)[None, :, None] * (1.0 + 0.1 * rng.random(U.shape))
    V *= (d * d)[None, :, None]
    W *= dg[None, :, None]
    got, ref = _nu_t(case, U, V, W)
    for j in range(case.Ny):
        assert np.abs(got[:, j] - ref[:, j]).max() <= NUT_RTOL * np.abs(ref[:, j]).max(), j
