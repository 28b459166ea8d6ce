"""The planner on a batch of one render: it reports a block that is launched."""
import pytest

from gray_b200 import api, configs


@pytest.mark.gpu
@pytest.mark.parametrize("n_freq", [0, 4])
def test_plan_of_one_render(ctx, n_freq):
    """The unrolled one-ray kernel of a single render has blocks of 128 threads
    at most; asked several times, since two equal shapes win by chance."""
    cfg = dict(configs.TORUS_RT_1024, n_width=192, n_height=128, r_obs=60.0, n_sub=200, n_dump=2,
               precision=api.PREC_MIXED)
    cfg["nu"] = cfg["nu"][:n_freq]
    r = ctx.render(cfg)
    b = ctx.batch([r])
    old = ctx.get_plan()
    try:
        for _ in range(8):
            p = ctx.plan(b, api.PLAN_MEASURE)
            assert p.block <= 128 or p.rk4_rolled == 1
            cur = ctx.get_plan()
            assert (cur.block, cur.blocks_per_sm) == (p.block, p.blocks_per_sm)
    finally:
        ctx.set_plan(old.block, old.blocks_per_sm, old.rays_per_thread, old.rk4_rolled)
        b.close()
        r.close()
