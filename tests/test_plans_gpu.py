"""Plans that depend on the batch: planes per thread and the remainders they
leave, rows per lane, and the step graph's side branch against the same kernels
in order."""
from dataclasses import replace

import numpy as np
import pytest

from channel_rl_gb300 import cases as C
from tests.helpers import FIELD_RTOL, oracle_for, regions, rel

pytestmark = pytest.mark.gpu

MODELS = (C.LES_NONE, C.LES_SMAG, C.LES_DSM, C.LES_AMD, C.LES_VREMAN)


def _fields(ch, q=0):
    d = ch.download(inst=q, fields=("U", "V", "W", "nu_t"))
    return [d[k] for k in ("U", "V", "W", "nu_t")] + list(ch.compute_rhs(q))


# twelve channels take four planes per thread in the marching kernels and 8 or 16
# in the test filter, one alone one plane and four: 18 and 54 leave two over, 20 four
@pytest.mark.parametrize("les", MODELS)
@pytest.mark.parametrize("wm", (C.WM_NONE, C.WM_EQLOG))
def test_planes_left_over_in_a_batch(les, wm):
    from channel_rl_gb300.host import Channel
    shapes = ((64, 41, 18), (54, 16, 54), (96, 33, 18), (36, 24, 54)) * 3
    batch = [replace(C.wallmodelled(f"b{n}", *s, 2000.0, les=les, wall_model=wm, seed=n), x_mass_cte=n % 2)
             for n, s in enumerate(shapes)]
    fields = [C.initial_fields(c) for c in batch]
    ch = Channel(batch)
    for q, f in enumerate(fields):
        ch.upload(*f, inst=q)
    ch.step(2)
    got = [_fields(ch, q) for q in range(4)]
    ch.close()
    for q in range(4):
        one = Channel(batch[q])
        one.upload(*fields[q])
        one.step(2)
        assert all(np.array_equal(a, b) for a, b in zip(got[q], _fields(one))), q
        one.close()


@pytest.mark.parametrize("les", MODELS)
@pytest.mark.parametrize("wm", (C.WM_NONE, C.WM_STRESS, C.WM_EQLOG, C.WM_MLP))
def test_the_step_graph_is_the_kernels_in_order(les, wm):
    """compute_dt and compute_time_step_RK3 issue on one stream what the graph's
    two branches run beside each other."""
    from channel_rl_gb300.host import Channel
    case = C.wallmodelled("g", 48, 16, 36, 3000.0, les=les, wall_model=wm, x_mass_cte=1)
    out = []
    for graph in (True, False):
        ch = Channel(case)
        ch.upload(*C.initial_fields(case))
        if wm == C.WM_STRESS:
            ch.set_wall_stress(np.asfortranarray(np.full((case.nx, 2, case.nz + 1), case.dPdx)))
        if wm == C.WM_MLP:
            ch.mlp_configure(sigma=0.1, seed=3, train=False)
        for _ in range(3):
            if graph:
                ch.step(1)
            else:
                ch.compute_dt()
                ch.compute_time_step_RK3()
        d = ch.download(fields=("U", "V", "W", "nu_t"))
        out.append([d[k] for k in ("U", "V", "W", "nu_t")] + [np.array(list(ch.scalars().values()))])
        ch.close()
    assert all(np.array_equal(a, b) for a, b in zip(*out))


@pytest.mark.parametrize("les", MODELS)
@pytest.mark.parametrize("wm", (C.WM_NONE, C.WM_EQLOG))
@pytest.mark.parametrize("bad", (np.nan, np.inf))
def test_a_non_finite_velocity_is_flagged(les, wm, bad):
    from channel_rl_gb300.host import Channel, ChlError
    case = C.wallmodelled("n", 16, 12, 16, 2000.0, les=les, wall_model=wm)
    for field, at in ((0, (5, 1, 7)), (1, (5, 6, 7)), (2, (9, 6, 3))):
        f = [a.copy(order="F") for a in C.initial_fields(case)]
        f[field][at] = bad
        ch = Channel(case)
        ch.upload(*f)
        ch.compute_eddy_viscosity()
        if wm:
            ch.compute_wall_model()
        F = ch.compute_rhs()
        assert not all(np.isfinite(a).all() for a in F)
        ch.step(1)
        with pytest.raises(ChlError):
            ch.synchronize()
        ch.upload(*C.initial_fields(case))          # nothing of it stays behind
        ch.step(1)
        ch.synchronize()
        assert all(np.isfinite(a).all() for a in ch.download().values())
        ch.close()


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
