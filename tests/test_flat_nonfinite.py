"""Rays with NaN or infinite coordinates outside a numerical spacetime's box
(gray_write_state takes any state): the mixed kernel ends such a ray at its
first step, and the rays beside it take theirs."""
import numpy as np
import pytest

from gray_b200 import api

CFG = dict(spacetime=api.ST_NUMERICAL, a_spin=0.0, i_obs=50.0, j_obs=20.0, w_img=24.0, h_img=24.0,
           n_width=9, n_height=1, r_obs=70.0, dt_dump=-3.0, n_dump=2, n_sub=100, precision=api.PREC_MIXED)


@pytest.mark.gpu
@pytest.mark.parametrize("row", [0, 1, 3])
@pytest.mark.parametrize("value", [np.nan, np.inf, 1e39])
def test_the_ray_ends_at_its_first_step(ctx, row, value):
    """1e39 is beyond FP32, in which the position is held."""
    ctx.make_boosted_ks(api.make_grid(20, -40.0, 40.0, physics=True), 0.7, 0.3, 1, 0.0, 0)
    r = ctx.render(CFG)
    try:
        r.icond()
        start = r.state()[0]
        r.evolve_all()
        want, per_ray = r.state()[0], r.steps() // 9
        bad = start.copy()
        bad[row, 4] = value
        r.icond()
        r.write_state(bad)
        r.evolve_all()
        got = r.state()[0]
        assert r.steps() == 8 * per_ray + 1
        others = np.arange(9) != 4
        assert np.array_equal(got[:, others], want[:, others])
        # the components the value does not touch have taken one step
        dt = -0.01
        for k in range(4):
            if k != row:
                moved = got[k, 4] - start[k, 4]
                assert abs(moved - dt * start[4 + k, 4]) <= 1e-6 * abs(dt) + 1e-12 * abs(start[k, 4])
    finally:
        r.close()
