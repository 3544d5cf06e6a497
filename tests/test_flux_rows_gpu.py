"""The right-hand side next to resolved walls, row by row: V falls as the square
of the wall distance and U as the distance, so a row's values are small beside
the field's largest, and each row has to keep its own digits."""
from dataclasses import replace

import numpy as np
import pytest

from channel_rl_gb300 import cases as C

pytestmark = pytest.mark.gpu
L = np.longdouble


def _rhs(case, U, V, W):
    """F of no model in extended precision from fields (z, y, x) on the unique
    points, and the sum of the magnitudes that its rounding errors scale with."""
    x, y, z = (a.astype(L) for a in C.faces(case))
    yg = C.centres_y(C.faces(case)[1]).astype(L)
    n, m, nu = case.Nx, case.Nz, L(case.nu)
    mid = lambda f: (f[:-1] + f[1:]) / 2
    per = lambda d, N: np.concatenate([d, d[:1]])[:N]      # spacing of the centres around a face
    xm, zm = mid(x), mid(z)
    dxc, dxf, dzc, dzf = np.diff(x)[:n], per(np.diff(xm), n), np.diff(z)[:m], per(np.diff(zm), m)
    dzc, dzf = dzc[:, None, None], dzf[:, None, None]
    dyc, dyf = np.diff(y)[:, None], np.diff(yg)[:, None]
    w1 = (y - yg[:-1])[:, None] / dyf
    l, r = (lambda f: np.roll(f, 1, 2)), (lambda f: np.roll(f, -1, 2))
    b, t = (lambda f: np.roll(f, 1, 0)), (lambda f: np.roll(f, -1, 0))
    lo, hi = (lambda f: f[:, :-1]), (lambda f: f[:, 1:])
    face = lambda f: (1 - w1) * lo(f) + w1 * hi(f)
    Uc, Wc = U[:, 1:-1], W[:, 1:-1]

    def flux(grad, adv):
        return nu * grad - adv, nu * abs(grad) + abs(adv)
    ux = flux((Uc - l(Uc)) / dxc, ((Uc + l(Uc)) / 2) ** 2)
    vy = flux((hi(V) - lo(V)) / dyc, ((hi(V) + lo(V)) / 2) ** 2)
    wz = flux((Wc - b(Wc)) / dzc, ((Wc + b(Wc)) / 2) ** 2)
    uw = (Uc + t(Uc)) * (Wc + r(Wc)) / 4
    uz, wx = flux((t(Uc) - Uc) / dzf, uw), flux((r(Wc) - Wc) / dxf, uw)
    uv, vw = face(U) * (V + r(V)) / 2, face(W) * (V + t(V)) / 2
    uy, vx = flux((hi(U) - lo(U)) / dyf, uv), flux((r(V) - V) / dxf, uv)
    wy, vz = flux((hi(W) - lo(W)) / dyf, vw), flux((t(V) - V) / dzf, vw)

    def total(*parts):      # (flux high, flux low, spacing)
        F = sum((h[0] - q[0]) / d for h, q, d in parts)
        return F, sum((h[1] + q[1]) / d for h, q, d in parts)
    up = lambda f, g: tuple(g(a) for a in f)
    i = lambda f: tuple(a[:, 1:-1] for a in f)
    Fu, Mu = total((up(ux, r), ux, dxf), (up(uy, hi), up(uy, lo), dyc), (uz, up(uz, b), dzc))
    Fv, Mv = total((i(vx), up(i(vx), l), dxc), (up(vy, hi), up(vy, lo), dyf[1:-1]), (i(vz), up(i(vz), b), dzc))
    Fw, Mw = total((wx, up(wx, l), dxc), (up(wy, hi), up(wy, lo), dyc), (up(wz, t), wz, dzf))
    return (Fu + L(case.dPdx), Fv, Fw), (Mu + abs(L(case.dPdx)), Mv, Mw)


@pytest.mark.parametrize("shape,stretch", (((16, 24, 12), 2.5), ((18, 48, 8), 3.0), ((8, 9, 6), 1.5)))
def test_rows_next_to_a_resolved_wall_keep_their_digits(shape, stretch):
    """Tolerance: eight FP64 roundings of the fluxes, spacings and differences that
    F of a row is made of."""
    from channel_rl_gb300.host import Channel
    case = replace(C.smaller(C.c1_small(), *shape), stretch=stretch, LES_model=C.LES_NONE, x_mass_cte=0, dPdx=1e-3)
    U, V, W = (a.copy(order="F") for a in C.initial_fields(case))
    d, dg = (1.0 - np.abs(y) for y in (C.faces(case)[1], C.centres_y(C.faces(case)[1])))
    rng = np.random.default_rng(5)
    U *= 0
    U += (1.5 * dg)[None, :, None] * (1.0 + 0.1 * rng.random(U.shape))
    V *= (d * d)[None, :, None]
    W *= dg[None, :, None]
    ch = Channel(case)
    ch.upload(U, V, W)
    ch.compute_eddy_viscosity()
    F = ch.compute_rhs()
    f = ch.download()
    ch.close()
    cut = {"U": (slice(1, case.Nx + 1), slice(1, case.Nz + 1)), "V": (slice(1, case.Nx + 1), slice(1, case.Nz + 1)),
           "W": (slice(1, case.Nx + 1), slice(1, case.Nz + 1))}
    fields = [np.ascontiguousarray(f[q][cut[q][0], :, cut[q][1]].T).astype(L) for q in "UVW"]
    ref, mag = _rhs(case, *fields)
    for got, e, m in zip(F, ref, mag):
        err = np.abs(got.T.astype(L) - e).max((0, 2))
        assert (err <= 8 * 2.0 ** -53 * m.max((0, 2))).all(), (err / m.max((0, 2)) * 2.0 ** 53).tolist()
