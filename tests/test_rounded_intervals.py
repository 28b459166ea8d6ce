"""Dump intervals whose ends round to the same time: t_init + i dt_dump in
FP64 need not move with i.  Such an interval has no step count (driver.cl:93
divides by its length); it leaves the state as it is, as evolving from t to t
does, and the intervals around it are walked."""
import numpy as np
import pytest

from gray_b200 import api, configs

KERR = dict(configs.TORUS_RT_1024, n_width=7, n_height=5, r_obs=40.0, n_sub=100)
NUM = dict(spacetime=api.ST_NUMERICAL, a_spin=0.0, i_obs=50.0, j_obs=20.0, w_img=24.0, h_img=24.0,
           n_width=7, n_height=5, r_obs=25.0, n_sub=100, nu=(2.3e11,), flow_te=1e3, flow_b=20.0)
ALL = dict(t_init=1e17, dt_dump=-1.0, n_dump=5)             # no interval has a length
SOME = dict(t_init=2.0**53 + 4.0, dt_dump=-1.0, n_dump=7)   # lengths 0, 2, 0, 2, then 1
INF = dict(t_init=1e308, dt_dump=1e308, n_dump=3)           # one of infinite length, then inf - inf


def setup(ctx, kind):
    if kind == "kerr":
        return KERR
    ctx.make_boosted_ks(api.make_grid(20, -40.0, 40.0), 0.7, 0.3, 1, 0.0, 0)
    return NUM


def lengths(c):
    t = [c["t_init"] + i * c["dt_dump"] for i in range(c["n_dump"] + 1)]
    return list(zip(t[:-1], t[1:]))


def test_the_cases_are_what_they_say():
    assert all(a == b for a, b in lengths(ALL))
    d = [b - a for a, b in lengths(SOME)]
    assert 0.0 in d and -2.0 in d and -1.0 in d


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [api.PREC_FP64, api.PREC_MIXED])
@pytest.mark.parametrize("kind", ["kerr", "numerical"])
@pytest.mark.parametrize("window", [ALL, SOME, INF], ids=["all", "some", "infinite"])
def test_run_equals_its_intervals(ctx, kind, precision, window):
    """Against one call per interval, which skips the empty ones: the same bits
    in FP64.  A mixed state passes HBM between calls and may come back split
    into another FP32 pair, which changes a step's increments by 2^-24: at
    most 2^-24 of the path (9 M) and of what is emitted, times the tens of
    operations of a right-hand side."""
    c = dict(setup(ctx, kind), precision=precision, **window)
    r = ctx.render(c)
    try:
        r.icond()
        for t, target in lengths(c):
            if t != target and np.isfinite(target - t):
                r.evolve(t, target)
        want = r.state()[0]
        steps = r.steps()
        r.run()
        got = r.state()[0]
        assert r.steps() == steps
    finally:
        r.close()
    if precision == api.PREC_FP64:
        assert np.array_equal(got, want)
    else:
        for row in range(8):
            assert np.linalg.norm(got[row] - want[row]) <= 1e-6 * np.linalg.norm(want[:8])
        for row in range(8, len(want)):
            assert np.linalg.norm(got[row] - want[row]) <= 1e-5 * np.linalg.norm(want[row])


@pytest.mark.gpu
def test_batch_skips_them(ctx):
    """Renders with and without such intervals in one launch, one ray and two
    per thread, the two-ray kernel's slots apart."""
    cfgs = [dict(KERR, precision=api.PREC_MIXED, **w) for w in (ALL, SOME, dict(n_dump=2))]
    old = ctx.get_plan()
    try:
        for plan in ((256, 0, 1, 0), (128, 0, 2, 0)):
            ctx.set_plan(*plan)
            rs = [ctx.render(c) for c in cfgs]
            b = ctx.batch(rs)
            try:
                b.run()
                got = [r.state()[0] for r in rs]
                for r, d in zip(rs, got):
                    r.run()
                    assert np.array_equal(r.state()[0], d)
                rs[0].icond()
                assert np.array_equal(rs[0].state()[0], got[0])
            finally:
                b.close()
                for r in rs:
                    r.close()
    finally:
        ctx.set_plan(old.block, old.blocks_per_sm, old.rays_per_thread, old.rk4_rolled)
