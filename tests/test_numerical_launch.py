"""Which launch a numerical render takes: the level rule reads the rays' own
time, so traces that differ only in the label of their affine time take the
same launch, and the launch never changes a result."""
import numpy as np
import pytest

from gray_b200 import api

BOX = 40.0
NU = (2.3e11, 8.6e10, 3.45e11)
BASE = dict(spacetime=api.ST_NUMERICAL, a_spin=0.0, i_obs=50.0, j_obs=20.0, w_img=24.0, h_img=24.0,
            r_obs=30.0, n_sub=100, flow_te=1e3, flow_b=20.0, precision=api.PREC_MIXED)


def grid(ctx, n, t1, t2, physics=True):
    g = api.make_grid(n, -BOX, BOX, t1, t2, physics=physics)
    ctx.make_boosted_ks(g, 0.7, 0.3, 1, t1, 0)
    if t2 != t1:
        ctx.make_boosted_ks(g, 0.7, 0.3, 1, t2, 1)


def ms(ctx, cfg):
    """The best of several runs, on the device."""
    r = ctx.render(cfg)
    try:
        return min(r.run() for _ in range(5)) * 1e-6
    finally:
        r.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nu", [(), NU], ids=["geodesics", "thermal"])
@pytest.mark.parametrize("t1,t2,label", [(-10.0, 0.0, 64.0),   # between the levels
                                         (0.0, 10.0, 10.0)])   # on the first one
def test_label_of_the_time_does_not_change_the_launch(ctx, nu, t1, t2, label):
    """The wrong launch takes twice to five times as long; the same one
    repeats within a few percent."""
    grid(ctx, 64, t1, t2)
    cfg = dict(BASE, nu=nu, n_width=300, n_height=200, dt_dump=-2.0, n_dump=5)
    a, b = ms(ctx, dict(cfg, t_init=0.0)), ms(ctx, dict(cfg, t_init=label))
    assert max(a, b) <= 1.25 * min(a, b), (a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("nu", [(), NU], ids=["geodesics", "thermal"])
def test_either_launch_gives_the_same_bits(ctx, nu):
    """Intervals called for another time than the rays': the one-level launch
    reads both levels directly, the two-level one holds a level without weight."""
    for t1, t2, t in ((-6.0, -1.0, 64.0), (0.0, 5.0, 4.0)):
        grid(ctx, 24, t1, t2)
        r = ctx.render(dict(BASE, r_obs=25.0, nu=nu, n_width=13, n_height=5, dt_dump=-2.0, n_dump=4, t_init=0.0))
        try:
            out = []
            for at in (0.0, t):
                r.icond()
                for i in range(4):
                    r.evolve(at - 2.0 * i, at - 2.0 * (i + 1))
                out.append(r.state()[0])
        finally:
            r.close()
        assert np.array_equal(out[0], out[1])


@pytest.mark.gpu
@pytest.mark.parametrize("nu", [(), NU], ids=["geodesics", "thermal"])
def test_rays_past_the_levels_keep_their_cells(ctx, nu):
    """A forward trace after the second level's time reads that level alone, as
    one on a single level does: the same steps in the same time (it took 1.3 to
    1.9 times as long while each step searched its cell), and the FP64
    kernel's result."""
    cfg = dict(BASE, r_obs=25.0, nu=nu, n_width=300, n_height=200, dt_dump=1.0, n_dump=8)
    grid(ctx, 64, -10.0, -1.0)
    past = ms(ctx, cfg)
    small = dict(cfg, n_width=13, n_height=5)
    out = []
    for precision in (api.PREC_FP64, api.PREC_MIXED):
        r = ctx.render(dict(small, precision=precision))
        r.run()
        out.append(r.state()[0])
        r.close()
    for row in range(1, 8):
        assert np.linalg.norm(out[1][row] - out[0][row]) <= 1e-4 * np.linalg.norm(out[0][:8])
    grid(ctx, 64, -1.0, -1.0)
    assert past <= 1.2 * ms(ctx, cfg)


@pytest.mark.gpu
def test_plan_blocks_keep_their_warps(ctx):
    """A plan of one 256-thread block per SM is eight warps in this kernel's
    128-thread blocks too (four took 1.6 times as long)."""
    grid(ctx, 64, 0.0, 0.0)
    cfg = dict(BASE, n_width=300, n_height=200, dt_dump=-2.0, n_dump=5)
    old = ctx.get_plan()
    try:
        ctx.set_plan(128, 2, 1)
        two = ms(ctx, cfg)
        ctx.set_plan(256, 1, 1)
        one = ms(ctx, cfg)
    finally:
        ctx.set_plan(old.block, old.blocks_per_sm, old.rays_per_thread, old.rk4_rolled)
    assert one <= 1.2 * two, (one, two)
