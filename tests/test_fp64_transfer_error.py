"""The FP64 torus transfer's rounding: one step so short that no event moves,
from states over the torus, against the same transfer in 80-bit floats.  The
kernel shares factors and exponentials; its mean error may not exceed that of
the same formulas written with the operators, pow and exp (the CPU oracle)."""
import numpy as np
import pytest

import oracle as O
from gray_b200 import api, configs

LD = np.longdouble
NU = (1.0, 2.0, 4.0, 8.0)
CFG = dict(configs.TORUS_RT_1024, nu=NU, n_width=128, n_height=96, n_sub=1, n_dump=1, dt_dump=-1e-30)
N = 128 * 96


def states(rng, a, zmax, taumax):
    """Events outside the ISCO with null u, as (16, N)."""
    risco = O.risco(a)
    r = risco * np.exp(rng.uniform(0.02, np.log(200.0), N))
    ct, ph = rng.uniform(-zmax, zmax, N), rng.uniform(0.0, 2.0 * np.pi, N)
    R = np.sqrt((r * r + a * a) * (1.0 - ct * ct))
    s = np.zeros((16, N))
    s[1], s[2], s[3] = R * np.cos(ph), R * np.sin(ph), r * ct
    d = rng.standard_normal((3, N))
    d /= np.linalg.norm(d, axis=0)
    f, l, _, _ = ks(a, s)
    ld = (l * d).sum(0)
    A, B, C = 1.0 + f * ld * ld, 2.0 * f * ld, f - 1.0
    s[4], s[5:8] = 1.0, d * ((-B + np.sqrt(B * B - 4.0 * A * C)) / (2.0 * A)).astype(float)
    s[12:16] = rng.uniform(0.0, taumax, (4, N))
    return s


def ks(a, s):
    x, y, z = (s[i].astype(LD) for i in (1, 2, 3))
    a = LD(a)
    k = (x * x + y * y + z * z - a * a) / 2
    rr = k + np.sqrt(k * k + a * a * z * z)
    r = np.sqrt(rr)
    f = 2 * rr * r / (rr * rr + a * a * z * z)
    iss = 1 / (rr + a * a)
    return f, np.stack([iss * (r * x + a * y), iss * (r * y - a * x), z / r]), r, iss


def exact(c, s):
    """dI, dtau (8, N) of the state in 80 bits."""
    a = LD(c["a_spin"])
    f, l, r, iss = ks(a, s)
    x, y, z, u = s[1].astype(LD), s[2].astype(LD), s[3].astype(LD), s[4:8].astype(LD)
    flu = f * (u[0] + (l * u[1:]).sum(0))
    kt, kx, ky = flu - u[0], u[1] + flu * l[0], u[2] + flu * l[1]
    R2 = x * x + y * y
    Om = 1 / (r * np.sqrt(r) + a)
    lv = 1 - a * Om * R2 * iss
    D = 1 - Om * Om * R2 - f * lv * lv
    sh = -(kt + Om * (x * ky - y * kx)) / np.sqrt(np.where(D > 0, D, 1))
    q = LD(O.rplus(c["a_spin"])) / r
    h = LD(c["torus_hr"]) * r
    n = LD(c["torus_n0"]) * q * np.sqrt(q) * np.exp(-z * z / (2 * h * h))
    ok = (D > LD(0.01)) & (sh > 0)      # a Keplerian flow near light speed amplifies every rounding
    sh = np.where(ok, sh, 1)
    nupow = np.array([float(v) ** -0.7 for v in NU]).astype(LD)[:, None]
    nuinv2 = np.array([1.0 / (v * v) for v in NU]).astype(LD)[:, None]
    dI = -n * sh ** LD(-0.7) * nupow * np.exp(-s[12:16].astype(LD)) / (sh * sh)
    dT = -(LD(c["torus_kappa"]) * n / sh) * nuinv2
    return dI, dT, ok


def step(ctx, c, s):
    r = ctx.render(dict(c, precision=api.PREC_FP64))
    try:
        r.icond()
        r.write_state(s)
        r.evolve_all()
        return r.state()[0]
    finally:
        r.close()


def oracle_step(c, s):
    return np.stack([O.integrate(c, s[:, i], c["dt_dump"]) for i in range(N)], axis=1)


@pytest.mark.gpu
@pytest.mark.parametrize("a_spin", [0.0, 0.9])
@pytest.mark.parametrize("zmax,taumax", [(0.1, 0.5), (0.5, 10.0), (1.0, 5.0)])
def test_no_larger_than_the_operators(ctx, a_spin, zmax, taumax):
    """I grows by dt dI (tau by dt dtau, from 0) through the same RK4 sum on both
    sides: 12,288 events, 49,152 values a mean."""
    rng = np.random.default_rng(17)
    c = dict(CFG, a_spin=a_spin)
    s = states(rng, a_spin, zmax, taumax)
    dt = LD(c["dt_dump"])
    dI, dT, ok = exact(c, s)
    assert ok.mean() > 0.5
    s0 = s.copy()
    s0[12:16] = 0.0
    gI, oI = (f[8:12].astype(LD) / dt for f in (step(ctx, c, s), oracle_step(c, s)))
    gT, oT = (f[12:16].astype(LD) / dt for f in (step(ctx, c, s0), oracle_step(c, s0)))

    def mean(v, want):
        return float(np.mean(np.abs((v[:, ok] - want[:, ok]) / want[:, ok]))) * 2.0**53

    eI, eT, wI, wT = mean(gI, dI), mean(gT, dT), mean(oI, dI), mean(oT, dT)
    print("dI %.3f (operators %.3f)  dtau %.3f (%.3f)" % (eI, wI, eT, wT))
    assert eI <= wI and eT <= wT
