"""The FP64 kernel's radius and quotients start from shared approximations;
rays from the far field to the horizon must still round like the oracle."""
import numpy as np
import pytest

import oracle as O
from gray_b200 import api, configs


@pytest.mark.gpu
@pytest.mark.parametrize("a_spin", [0.0, 0.5, 0.998, -0.9])
@pytest.mark.parametrize("i_obs,r_obs", [(5.0, 40.0), (90.0, 25.0), (60.0, 1e5)])
def test_geodesics_round_like_the_oracle(ctx, a_spin, i_obs, r_obs):
    """Bit for bit, captured rays among them: the oracle's divides and roots
    are rounded to nearest, and so are the kernel's (one ulp is left where a
    divisor's significand is all ones: 1 in 2^52 quotients)."""
    cfg = dict(configs.KERR_SMALL_64, a_spin=a_spin, i_obs=i_obs, r_obs=r_obs, n_width=12, n_height=9,
               w_img=14.0, h_img=14.0, n_dump=2)
    r = ctx.render(dict(cfg, precision=api.PREC_FP64))
    try:
        r.run()
        got, _ = r.state(api.LAYOUT_AOS)
        steps = r.steps()
    finally:
        r.close()
    ref, _, n = O.trace(cfg, np.arange(12 * 9))
    assert steps == n.sum()
    assert np.array_equal(got, ref)
