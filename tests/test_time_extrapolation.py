"""Outside the levels' times in reference semantics (no physics box) the
fields extrapolate linearly in time (interp.cl:183-205): the mixed kernel
against the FP64 kernel, which the CPU oracle pins."""
import numpy as np
import pytest

from gray_b200 import api

BOX = 40.0
CFG = dict(spacetime=api.ST_NUMERICAL, a_spin=0.0, i_obs=50.0, j_obs=20.0, w_img=24.0, h_img=24.0,
           n_width=13, n_height=5, r_obs=25.0, n_sub=100, flow_te=1e3, flow_b=20.0)


def state(ctx, cfg):
    r = ctx.render(cfg)
    try:
        r.run()
        return r.state()[0], r.steps()
    finally:
        r.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nu", [(), (2.3e11, 8.6e10, 3.45e11)], ids=["geodesics", "thermal"])
@pytest.mark.parametrize("t1,t2,over", [
    (-9.0, -4.0, dict(dt_dump=-2.0, n_dump=2)),   # after the levels alone
    (1.0, 5.0, dict(dt_dump=-2.0, n_dump=4)),     # before them alone, far below
    (-5.0, -2.0, dict(dt_dump=-2.0, n_dump=4)),   # after, between, before
    (-3.0, 0.0, dict(dt_dump=2.0, n_dump=3)),     # forward from the last level
])
def test_mixed_extrapolates(ctx, nu, t1, t2, over):
    """At most 800 steps; the extrapolated sums (1 - ft) L0 + ft L1 carry the
    rounding of terms up to 9/4 and 5/4 the fields, so the bound of a trace
    between the levels (a relative 2^-24 per operation on increments that sum
    to the path, 1e-4 of the state's norm at most) holds here too."""
    g = api.make_grid(24, -BOX, BOX, t1, t2)
    ctx.make_boosted_ks(g, 0.7, 0.3, 1, t1, 0)
    ctx.make_boosted_ks(g, 0.7, 0.3, 1, t2, 1)
    cfg = dict(CFG, nu=nu, **over)
    ref, s64 = state(ctx, dict(cfg, precision=api.PREC_FP64))
    got, smx = state(ctx, dict(cfg, precision=api.PREC_MIXED))
    assert smx == s64 and np.isfinite(ref).all() and np.isfinite(got).all()
    start = ctx.render(dict(cfg, precision=api.PREC_FP64))
    start.icond()
    u0 = start.state()[0][4:8]
    start.close()
    # what the spacetime did to u, not u itself, is what is compared
    assert np.linalg.norm(got[4:8] - ref[4:8]) <= 1e-3 * np.linalg.norm(ref[4:8] - u0)
    for rows in (slice(0, 4), slice(4, 8)) + tuple(slice(8 + i, 9 + i) for i in range(2 * len(nu))):
        assert np.linalg.norm(got[rows] - ref[rows]) <= 1e-4 * np.linalg.norm(ref[rows])
