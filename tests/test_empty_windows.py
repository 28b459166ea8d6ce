"""Renders without dump intervals ahead of others in one launch: their rays
hand their lanes straight back, and the rays queued behind them are traced."""
import numpy as np
import pytest

from gray_b200 import api, configs

BASE = dict(configs.TORUS_RT_1024, r_obs=40.0, n_sub=100, precision=api.PREC_MIXED)


@pytest.mark.gpu
@pytest.mark.parametrize("n_freq", [0, 4])
@pytest.mark.parametrize("plan", [(256, 0, 1, 0), (256, 0, 1, 1), (128, 0, 2, 0)],
                         ids=["one", "rolled", "two"])
def test_rays_behind_empty_windows_are_traced(ctx, plan, n_freq):
    """900 x 900 empty rays are more than the device holds at once (148 SMs of
    2,048 threads, two rays each), so every warp draws some first."""
    base = dict(BASE, nu=BASE["nu"][:n_freq])
    cfgs = [dict(base, n_width=900, n_height=900, n_dump=0),
            dict(base, n_width=13, n_height=7, n_dump=2),
            dict(base, n_width=33, n_height=1, n_dump=0),
            dict(base, n_width=5, n_height=3, n_dump=1)]
    old = ctx.get_plan()
    try:
        ctx.set_plan(*plan)
        rs = [ctx.render(c) for c in cfgs]
        b = ctx.batch(rs)
        try:
            b.run()
            got = [r.state() for r in rs]
            steps = b.steps()
            want_steps = 0
            for r, (d, info), c in zip(rs, got, cfgs):
                if c["n_dump"]:
                    r.run()
                    want_steps += r.steps()
                else:
                    r.icond()
                want, winfo = r.state()
                assert np.array_equal(d, want)
                assert c["n_dump"] == 0 or np.array_equal(info, winfo)
            assert steps == want_steps > 0
        finally:
            b.close()
            for r in rs:
                r.close()
    finally:
        ctx.set_plan(old.block, old.blocks_per_sm, old.rays_per_thread, old.rk4_rolled)
