"""Runs of capped steps far from the hole: the mixed kernel takes them without
asking the step rule, and must take the ones the rule would."""
import numpy as np
import pytest

from gray_b200 import api, configs

BASE = dict(configs.TORUS_RT_1024, n_width=13, n_height=7, a_spin=0.8, i_obs=55.0)


def run(ctx, cfg, precision):
    r = ctx.render(dict(cfg, precision=precision))
    try:
        r.run()
        return r.state()[0], r.steps()
    finally:
        r.close()


@pytest.mark.gpu
@pytest.mark.parametrize("cfg", [
    dict(r_obs=1000.0, n_dump=2),                             # whole intervals at once
    dict(r_obs=60.0, n_dump=3, dt_dump=-17.3, n_sub=701),     # a last step that is not whole
    dict(r_obs=60.0, n_dump=2, dt_dump=-0.05, n_sub=3),       # fewer steps than are asked for
    dict(r_obs=25.0, n_dump=2, dt_dump=8.0, n_sub=400, nu=()),  # forward, away from the hole
])
def test_capped_runs_match_fp64(ctx, cfg):
    """No ray comes within the region where the step is shorter than the cap,
    so the counts are equal; at most 4,000 compensated steps add 2^-24 each
    to increments that sum to the path: 1e-4 of the state (the project's
    image bound) is far above that."""
    cfg = dict(BASE, **cfg)
    ref, s64 = run(ctx, cfg, api.PREC_FP64)
    got, smx = run(ctx, cfg, api.PREC_MIXED)
    assert smx == s64
    for rows in (slice(0, 4), slice(4, 8)) + tuple(slice(8 + i, 9 + i) for i in range(2 * len(cfg["nu"]))):
        assert np.linalg.norm(got[rows] - ref[rows]) <= 1e-4 * np.linalg.norm(ref[rows])


@pytest.mark.gpu
def test_runs_do_not_depend_on_the_warp(ctx):
    """A ray's steps are the same whatever rays share its warp: rows of one
    image alone and together, captured rays among them."""
    cfg = dict(BASE, r_obs=40.0, n_dump=4, n_width=33, n_height=9, w_img=20.0, h_img=20.0,
               precision=api.PREC_MIXED)
    whole, _ = run(ctx, cfg, api.PREC_MIXED)
    w = cfg["n_width"]
    for row in (0, 4, 8):
        part, _ = run(ctx, dict(cfg, row_begin=row, n_rows=1), api.PREC_MIXED)
        assert np.array_equal(part, whole[:, row * w:(row + 1) * w])
