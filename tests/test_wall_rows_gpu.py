"""The rows next to a modelled wall, where nu + nu_t = tau dyw/du has no bound:
a wall point with nearly no shear may change only what lies beside it."""
from dataclasses import replace

import numpy as np
import pytest

from channel_rl_gb300 import cases as C
from tests.helpers import FIELD_RTOL, oracle_for

pytestmark = pytest.mark.gpu


# Ny = 8: the smallest with an equilibrium wall model; WM_STRESS from Ny = 5
@pytest.mark.parametrize("shape,wm", (((32, 16, 24), C.WM_EQLOG), ((18, 8, 12), C.WM_EQLOG), ((16, 5, 12), C.WM_STRESS)))
@pytest.mark.parametrize("shear", (1e-2, 1e-9, 0.0))
def test_a_point_without_wall_shear_moves_only_its_neighbours(shape, wm, shear):
    """F of every row at all other points, each row relative to its own largest
    there.  FIELD_RTOL: F is a sum of eighteen fluxes of at most a few hundred
    times its size, each with FP64 rounding."""
    from channel_rl_gb300.host import Channel
    case = replace(C.smaller(C.c2_wm64(), *shape), LES_model=C.LES_SMAG, wall_model=wm, x_mass_cte=0)
    U, V, W = (a.copy(order="F") for a in C.initial_fields(case))
    i0, k0 = 6, 7                                # Fortran index - 1 of the point, both walls
    U[i0, 1, k0] *= shear
    U[i0, -2, k0] *= shear
    o = oracle_for(case)
    o.set_fields(U, V, W)
    ch = Channel(case)
    ch.upload(U, V, W)
    if wm == C.WM_STRESS:
        a = np.asfortranarray(np.full((case.nx, 2, case.nz + 1), case.dPdx))
        ch.set_wall_stress(a)
        o.alpha_x[1:, 1:, 1:] = a
    ch.compute_eddy_viscosity()
    ch.compute_wall_model()
    F = ch.compute_rhs()
    ch.close()
    with np.errstate(all="ignore"):
        o._stage_sgs_wm()
        n, m = case.Nx, case.Nz
        ref = (o.compute_rhs_u(o.U, o.V, o.W, o.nu_t, o.dPdx)[:, :, :m], o.compute_rhs_v(o.U, o.V, o.W, o.nu_t)[:n, :, :m],
               o.compute_rhs_w(o.U, o.V, o.W, o.nu_t)[:n])
    far = np.ones((n, m), bool)
    far[i0 - 4:i0 + 4, k0 - 4:k0 + 3] = False
    for got, r in zip(F, ref):
        for j in range(r.shape[1]):
            g, e = got[:, j][far], r[:, j][far]
            assert np.isfinite(e).all() and np.abs(g - e).max() < FIELD_RTOL * np.abs(e).max(), j
