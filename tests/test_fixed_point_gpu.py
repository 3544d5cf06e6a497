"""The fixed-point kernels (momentum fluxes and transforms) where their scales
change: line lengths of every mix of radices, fields scaled by powers of two
(every exponent moves, no digit may), fields of very different magnitude, and
a non-finite value, which has to reach the result."""
from dataclasses import replace

import numpy as np
import pytest

from channel_rl_gb300 import cases as C
from tests.helpers import FIELD_RTOL, NUT_RTOL, oracle_for, regions, rel

pytestmark = pytest.mark.gpu

LENGTHS = ((4, 6), (6, 4), (8, 12), (12, 18), (24, 8), (54, 36), (32, 96), (48, 192), (256, 16), (162, 24), (16, 288), (1024, 4))


@pytest.mark.parametrize("Nx,Nz", LENGTHS)
def test_projection_of_every_radix_mix(Nx, Nz):
    """FIELD_RTOL: the transforms' rounding (2^-53 of a line's largest value
    per pass, as FP64's) passes to the gradient with factors of order one."""
    from channel_rl_gb300.host import Channel
    case = replace(C.smaller(C.c1_small(), Nx, 9, Nz), LES_model=C.LES_NONE, amp=1.0)
    U, V, W = C.initial_fields(case)
    o = oracle_for(case)
    o.set_fields(U, V, W)
    o.compute_projection_step()
    ch = Channel(case)
    ch.upload(U, V, W)
    ch.compute_projection_step()
    d = ch.download()
    reg = regions(o.g)
    for f in "UVW":
        r = reg[f][0], slice(1, -1), reg[f][2]      # the oracle leaves the ghost rows to the boundary conditions
        assert rel(d[f][r], getattr(o, f)[1:, 1:, 1:][r]) < FIELD_RTOL, f
    ch.close()


# the test filter's blocks: several x-lines, one line, a line cut into
# segments (more than 256 point pairs); one and two rows in the last group
@pytest.mark.parametrize("Nx,Ny,Nz", ((4, 8, 6), (6, 9, 4), (18, 6, 32), (256, 7, 6), (512, 6, 4), (576, 7, 4), (1024, 5, 4)))
def test_dynamic_model_over_line_lengths(Nx, Ny, Nz):
    from channel_rl_gb300.host import Channel
    case = C.smaller(C.c1_small(), Nx, Ny, Nz)
    U, V, W = C.initial_fields(case)
    o = oracle_for(case)
    o.set_fields(U, V, W)
    o.compute_eddy_viscosity()
    ch = Channel(case)
    ch.upload(U, V, W)
    ch.compute_eddy_viscosity()
    nt = ch.download(fields=("nu_t",))["nu_t"]
    ch.close()
    reg = regions(o.g)["C"]
    assert rel(nt[reg], o.nu_t[1:, 1:, 1:][reg]) < NUT_RTOL


def _rhs(case, U, V, W):
    from channel_rl_gb300.host import Channel
    ch = Channel(case)
    ch.upload(U, V, W)
    ch.compute_eddy_viscosity()
    F = ch.compute_rhs()
    nt = ch.download(fields=("nu_t",))["nu_t"]
    ch.compute_projection_step()
    d = ch.download()
    ch.close()
    return F, nt, d


@pytest.mark.parametrize("les", (C.LES_NONE, C.LES_SMAG, C.LES_DSM, C.LES_AMD, C.LES_VREMAN))
@pytest.mark.parametrize("k", (40, -44))
def test_powers_of_two_scale_through(les, k):
    """U, V, W, nu times 2^k and dPdx times 4^k: nu_t and the projected
    velocities times 2^k, F times 4^k, bit for bit (the static model's
    damping takes only ratios that do not change)."""
    s = 2.0 ** k
    case = replace(C.smaller(C.c1_small(), 18, 11, 12), LES_model=les, x_mass_cte=0, dPdx=0.01)
    big = replace(case, nu=case.nu * s, dPdx=case.dPdx * s * s)
    f = C.initial_fields(case)
    F, nt, d = _rhs(case, *f)
    Fs, nts, ds = _rhs(big, *(a * s for a in f))
    assert np.array_equal(nts, nt * s)
    for a, b in zip(Fs, F):
        assert np.array_equal(a, b * s * s)
    for q in "UVW":
        assert np.array_equal(ds[q], d[q] * s), q


def test_components_of_different_magnitude():
    """V and W 2^-30 of U: each component keeps its own scale, so V and W of
    the right-hand side agree with the oracle relative to themselves."""
    from channel_rl_gb300.host import Channel
    case = replace(C.smaller(C.c1_small(), 16, 12, 16), LES_model=C.LES_NONE)
    U, V, W = C.initial_fields(case)
    V, W = V * 2.0 ** -30, W * 2.0 ** -30
    o = oracle_for(case)
    o.set_fields(U, V, W)
    ch = Channel(case)
    ch.upload(U, V, W)
    ch.compute_eddy_viscosity()
    F = ch.compute_rhs()
    ch.close()
    o.compute_eddy_viscosity()
    n, m = case.Nx, case.Nz
    ref = (o.compute_rhs_u(o.U, o.V, o.W, o.nu_t, o.dPdx)[:, :, :m], o.compute_rhs_v(o.U, o.V, o.W, o.nu_t)[:n, :, :m],
           o.compute_rhs_w(o.U, o.V, o.W, o.nu_t)[:n])
    for got, r in zip(F, ref):
        assert rel(got, r) < FIELD_RTOL


def test_a_non_finite_value_reaches_the_result():
    from channel_rl_gb300.host import Channel
    case = replace(C.smaller(C.c1_small(), 16, 12, 16), LES_model=C.LES_AMD)
    for bad in (np.nan, np.inf):
        U, V, W = (a.copy(order="F") for a in C.initial_fields(case))
        V[5, 6, 7] = bad
        ch = Channel(case)
        ch.upload(U, V, W)
        ch.compute_eddy_viscosity()
        assert all(np.isnan(f).any() for f in ch.compute_rhs())
        ch.compute_projection_step()
        assert not np.isfinite(ch.pseudo_pressure()).all()
        ch.close()


# the mass-flow sum's blocks: one, several, as many as the partials have room for
@pytest.mark.parametrize("Nx,Nz", ((32, 16), (64, 32), (48, 64), (1024, 4), (2304, 4)))
def test_mass_flow_is_kept(Nx, Nz):
    from channel_rl_gb300.host import Channel
    case = replace(C.smaller(C.c1_small(), Nx, 8, Nz), LES_model=C.LES_NONE)
    U, V, W = C.initial_fields(case)
    o = oracle_for(case)
    o.set_fields(U, V, W)
    ch = Channel(case)
    ch.upload(U, V, W)
    reg = regions(o.g)["U"]
    for _ in range(2):                       # the second finds the block counter as the first left it
        o.step()
        ch.step(1)
        assert rel(ch.download(fields=("U",))["U"][reg], o.U[1:, 1:, 1:][reg]) < FIELD_RTOL
        assert abs(ch.compute_dPx_for_constant_mass_flow()) < 1e-12
    ch.close()
