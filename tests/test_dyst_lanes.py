"""The numerical kernels' lanes, cells and level codes: where a ray's cell,
box side or time levels change, and at the edges of its groups."""
import numpy as np
import pytest

import oracle as O
from gray_b200 import api

BOX = 40.0
NU = (2.3e11, 8.6e10, 3.45e11, 6.9e11, 4.3e10, 1.3e11, 1e12, 5e12)
BASE = dict(spacetime=api.ST_NUMERICAL, a_spin=0.0, i_obs=50.0, j_obs=20.0, w_img=24.0, h_img=24.0,
            r_obs=25.0, dt_dump=-2.0, n_sub=100, n_dump=4, flow_te=1e3, flow_b=20.0)


def grid_for(ctx, n, t1, t2, physics):
    g = api.make_grid(n, -BOX, BOX, t1, t2, physics=physics)
    ctx.make_boosted_ks(g, 0.7, 0.3, 1, t1, 0)
    if t2 != t1:
        ctx.make_boosted_ks(g, 0.7, 0.3, 1, t2, 1)


def state(ctx, cfg):
    r = ctx.render(dict(BASE, **cfg))
    try:
        r.run()
        return r.state()[0], r.steps()
    finally:
        r.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n_freq", [0, 1, 4, 5, 8])
@pytest.mark.parametrize("shape,n,levels,physics,cfg", [
    ((1, 1), 24, (0.0, 0.0), True, {}),                             # one ray in a warp
    ((9, 1), (2, 3, 5), (0.0, 0.0), False, {}),                     # fewest nodes: edge cells alone
    ((13, 5), 24, (-8.0, 0.0), False, {}),                          # eight lanes per ray
    ((13, 5), 24, (-5.0, -2.0), True, {}),                          # before, between and after the levels
    ((13, 5), 24, (0.0, 5.0), True, dict(r_obs=60.0, dt_dump=-10.0, n_dump=6)),  # into the box
])
def test_mixed_matches_fp64(ctx, n_freq, shape, n, levels, physics, cfg):
    """Over at most 6,000 steps of 0.01 M the FP32 right-hand side adds a
    relative 2^-24 per step and operation to increments that sum to the path
    (60 M): 60 x 6e-8 x tens of operations, 1e-4 of the state's norm at most
    (the project's image bound)."""
    grid_for(ctx, n, *levels, physics)
    cfg = dict(cfg, n_width=shape[0], n_height=shape[1], nu=NU[:n_freq])
    ref, s64 = state(ctx, dict(cfg, precision=api.PREC_FP64))
    got, smx = state(ctx, dict(cfg, precision=api.PREC_MIXED))
    assert np.isfinite(ref).all() and np.isfinite(got).all() and s64 == smx
    for rows in (slice(0, 4), slice(4, 8)) + tuple(slice(8 + i, 9 + i) for i in range(2 * n_freq)):
        assert np.linalg.norm(got[rows] - ref[rows]) <= 1e-4 * np.linalg.norm(ref[rows])


@pytest.mark.gpu
@pytest.mark.parametrize("n_freq", [0, 3])
def test_level_rule_does_not_change_results(ctx, n_freq):
    """A ray's time counts from the camera, so the same trace labelled with
    another t_init (which the launch rule reads) takes the one-level launch
    and its direct reads between the levels: the same bits."""
    grid_for(ctx, 24, -6.0, -1.0, True)
    cfg = dict(n_width=13, n_height=5, nu=NU[:n_freq], precision=api.PREC_MIXED)
    two, _ = state(ctx, dict(cfg, t_init=0.0))
    one, _ = state(ctx, dict(cfg, t_init=64.0))
    assert np.array_equal(one, two)


@pytest.mark.gpu
def test_chunked_flat_steps_keep_every_step(ctx):
    """Outside the box whole chunks of steps run at once: intervals that do
    not divide into whole steps, and one render's rays beside another's."""
    grid_for(ctx, 24, 0.0, 0.0, True)
    base = dict(precision=api.PREC_MIXED, n_width=7, n_height=3, r_obs=70.0, n_sub=33)
    cfgs = [dict(base, dt_dump=-7.003, n_dump=5), dict(base, dt_dump=-0.005, n_dump=3, r_obs=45.0),
            dict(base, dt_dump=-3.0, n_dump=9, n_sub=1000)]
    alone = [state(ctx, c) for c in cfgs]
    for c, (d, steps) in zip(cfgs, alone):
        ref, s64 = state(ctx, dict(c, precision=api.PREC_FP64))
        assert steps == s64
        assert np.linalg.norm(d - ref) <= 1e-6 * np.linalg.norm(ref)
    rs = [ctx.render(dict(BASE, **c)) for c in cfgs]
    b = ctx.batch(rs)
    try:
        b.run()
        for r, (d, _) in zip(rs, alone):
            assert np.array_equal(r.state()[0], d)
    finally:
        b.close()
        for r in rs:
            r.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n_freq", [0, 5])
@pytest.mark.parametrize("shape,levels,physics,cfg", [
    ((1, 1), (0.0, 0.0), True, dict(r_obs=45.0, dt_dump=-7.0, n_dump=2)),     # flat chunks, then the box
    ((9, 1), (0.0, 0.0), False, dict(r_obs=44.0, dt_dump=-3.0, n_dump=3)),    # clamped past the last node
    ((13, 5), (-3.0, 0.0), False, dict(n_dump=3)),                            # eight lanes per ray
    ((7, 3), (-3.0, -1.0), True, dict(n_dump=3, r_obs=41.0)),                 # time clamped at both ends
])
def test_fp64_lanes_match_oracle(ctx, n_freq, shape, levels, physics, cfg):
    """Each lane's operations are the oracle's in its order: the geodesic
    columns and step counts are equal, the transfer within 1e-10 (its exp,
    log and cbrt are not glibc's)."""
    n = 20
    t1, t2 = levels
    lv = [O.boosted_ks_grid(n, -BOX, BOX, t, a=0.7, v=0.3, axis=1) for t in levels]
    grid = api.make_grid(n, -BOX, BOX, t1, t2, physics=physics)
    for k in (0, 1):
        ctx.load_spacetime(grid, lv[k], k)
    og = O.Grid(lv if t1 != t2 else lv[:1], [t1, -BOX, -BOX, -BOX, t2, BOX, BOX, BOX],
                physics=physics)
    c = dict(BASE, **dict(cfg, n_width=shape[0], n_height=shape[1], nu=NU[:n_freq],
                          precision=api.PREC_FP64))
    got, steps = state(ctx, c)
    ref, _, osteps = O.dyst_trace(c, og, np.arange(shape[0] * shape[1]))
    assert steps == osteps.sum()
    assert np.array_equal(got[:8].T, ref[:, :8])
    assert np.all(np.abs(got[8:].T - ref[:, 8:]) <= 1e-10 * np.abs(ref[:, 8:]))
