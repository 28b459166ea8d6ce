"""The FP64 kernel's steps with the operators: rays beyond the range in which
its own quotients and roots hold (r^2 > 1e60), against the CPU oracle."""
import numpy as np
import pytest

import oracle as O
from gray_b200 import api, configs


@pytest.mark.gpu
@pytest.mark.parametrize("n_freq", [0, 1, 4, 8])
@pytest.mark.parametrize("r_obs", [0.5e30, 2e30, 1e31])   # one within the range
def test_rays_out_of_range_match_the_oracle(ctx, r_obs, n_freq):
    """Geodesics bit for bit; the transfer within the 1e-10 parity bar (its
    exp and pow are not glibc's)."""
    nu = (1.0, 2.0, 4.0, 8.0, 1.5, 3.0, 6.0, 12.0)[:n_freq]
    cfg = dict(configs.TORUS_RT_1024, a_spin=0.7, i_obs=80.0, r_obs=r_obs, n_width=7, n_height=5,
               w_img=r_obs, h_img=r_obs, dt_dump=-0.05 * r_obs, n_sub=50, n_dump=2, nu=nu)
    r = ctx.render(dict(cfg, precision=api.PREC_FP64))
    try:
        r.run()
        got, _ = r.state(api.LAYOUT_AOS)
        steps = r.steps()
    finally:
        r.close()
    ref, _, n = O.trace(cfg, np.arange(35))
    assert steps == n.sum() == 35 * 100
    assert np.array_equal(got[:, :8], ref[:, :8])
    if n_freq:
        # in the equatorial image row something is emitted; elsewhere the torus is thin
        assert (ref[:, 8:8 + n_freq] > 0).any()
        assert np.all(np.abs(got[:, 8:] - ref[:, 8:]) <= 1e-10 * np.abs(ref[:, 8:]))
