"""The work that a program using this framework has it do, as timed cases.

A case is one pass of a user's program: the call that renders (one image, a
batch of images, or one dump interval after another) and the read of the
rays' final state.  Kinds:

noalloc     gray_run_mixed_noalloc: renders into the caller's device buffers
render      Render.run + Render.state: a whole image of the analytic (Kerr)
            spacetime from its camera, in mixed or plain FP64 precision
dumps       the job's loop: icond, then evolve and read every dump interval
batch       many cameras of uneven sizes in one launch (Batch.run)
numerical   Render.run + Render.state on a resident numerical spacetime

Every render is made from the seed alone: spin, inclination and azimuth are
drawn over the ranges of the survey and serving workloads (a ~ U[0, 0.998],
inclination ~ U[5, 85] deg); step control, torus and image size are theirs.
A server runs the kernels of `batch` and `numerical` over windows of dump
intervals whose bounds depend on arrival times, so it is not timed here.
"""
import ctypes
import math
import random

import numpy as np
import torch

from gray_b200 import api, configs, flops

NU_TORUS = (1.0, 2.0, 4.0, 8.0, 1.5, 3.0, 6.0, 12.0)
NU_THERMAL = (2.3e11, 8.6e10, 3.45e11, 6.9e11, 4.3e10, 1.3e11, 1e12, 5e12)  # Hz
TE, B_FIELD = 1e3, 20.0                       # the thermal flow's kT/(m_e c^2) and field (G)
BOX = 40.0                                    # the numerical grids span [-BOX, BOX]^3
DT, N_SUB = -31.25, 1000                      # dump interval and substeps of the analytic workloads
LAYOUT = {"soa": api.LAYOUT_SOA, "aos": api.LAYOUT_AOS}


def listed():
    return [
        # the smallest call: two thumbnails near the hole, one frequency, into
        # buffers the caller owns (a preview, or one probe of a fit)
        dict(name="noalloc_thumbs", kind="noalloc", count=2, w=24, h=16, nf=1, r_obs=50.0, n_dump=1),
        # the smallest request of the serving mix: 64 x 64 at 1000 M, whole path
        dict(name="torus_64", kind="render", precision="mixed", w=64, h=64, nf=4, r_obs=1000.0, n_dump=64),
        # geodesics alone on an odd window of a camera at 300 M (lensing maps)
        dict(name="geodesics_333x187", kind="render", precision="mixed", w=333, h=187, nf=0, r_obs=300.0,
             n_dump=20),
        # the first dump interval of a large image near the hole
        dict(name="torus_512x384_near", kind="render", precision="mixed", w=512, h=384, nf=4, r_obs=40.0,
             n_dump=1),
        # the headline render
        dict(name="torus_1024", kind="render", precision="mixed", w=1024, h=1024, nf=4, r_obs=1000.0,
             n_dump=64),
        # a survey: cameras of uneven sizes, spins and distances in one launch
        dict(name="survey_24", kind="batch", count=24, lo=32, hi=256, nf=4, n_dump=64),
        # the plain FP64 job at its small size, dump by dump (kerr_small_64)
        dict(name="fp64_dumps_64", kind="dumps", precision="fp64", w=64, h=64, nf=0, r_obs=1000.0, n_dump=64,
             layout="aos"),
        # plain FP64 with transfer, an odd image through the hole's region
        dict(name="fp64_torus_251x190", kind="render", precision="fp64", w=251, h=190, nf=4, r_obs=100.0,
             n_dump=8),
        # the numerical spacetime at its workload's size
        dict(name="numerical_512", kind="numerical", precision="mixed", w=512, h=512, nf=0, grid=128,
             levels=2, physics=True, r_obs=200.0, dt=-10.0, n_dump=30),
        # a small numerical request of the serving mix on its 256^3 grid
        dict(name="numerical_97x72_grid256", kind="numerical", precision="mixed", w=97, h=72, nf=0, grid=256,
             levels=1, physics=True, r_obs=200.0, dt=-10.0, n_dump=30),
        # thermal transfer between two snapshots, camera inside the box
        dict(name="thermal_160x120", kind="numerical", precision="mixed", w=160, h=120, nf=4, grid=64,
             levels=2, physics=False, r_obs=30.0, dt=-2.0, n_dump=5),
        # the reference's own form: FP64, two snapshots, one frequency
        dict(name="numerical_fp64_64x48", kind="numerical", precision="fp64", w=64, h=48, nf=1, grid=64,
             levels=2, physics=False, r_obs=30.0, dt=-2.0, n_dump=5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("noalloc", "render", "render", "fp64", "dumps", "batch", "numerical", "numerical",
                       "thermal", "numerical_fp64"))
    robs = lambda lo, hi: round(math.exp(rng.uniform(math.log(lo), math.log(hi))), 3)  # noqa: E731
    if kind == "noalloc":
        return dict(kind="noalloc", count=rng.randint(1, 6), w=_log(rng, 8, 64), h=_log(rng, 8, 64),
                    nf=rng.randint(0, 4), r_obs=robs(45.0, 200.0), n_dump=rng.randint(1, 3))
    if kind in ("render", "fp64"):
        fp64 = kind == "fp64"
        w, h = _log(rng, 24, 256 if fp64 else 900), _log(rng, 24, 200 if fp64 else 700)
        r = robs(40.0, 150.0 if fp64 else 1000.0)
        # the whole path there and back, or its first intervals
        n = int(math.ceil(2 * r / -DT)) if rng.random() < 0.6 else rng.randint(1, 3)
        return dict(kind="render", precision="fp64" if fp64 else "mixed", w=w, h=h,
                    nf=rng.choice((0, 1, 2, 3, 4, 4, 8)), r_obs=r, n_dump=n)
    if kind == "dumps":
        return dict(kind="dumps", precision=rng.choice(("fp64", "mixed")), w=_log(rng, 16, 160),
                    h=_log(rng, 16, 120), nf=rng.choice((0, 0, 1, 4)), r_obs=robs(40.0, 300.0),
                    n_dump=rng.randint(2, 20), layout=rng.choice(("aos", "soa")))
    if kind == "batch":
        lo = _log(rng, 16, 64)
        return dict(kind="batch", count=rng.randint(2, 30), lo=lo, hi=lo * rng.choice((1, 2, 3, 4)),
                    nf=rng.choice((0, 1, 4)), n_dump=rng.randint(8, 64))
    if kind == "numerical":
        return dict(kind="numerical", precision="mixed", w=_log(rng, 24, 512), h=_log(rng, 24, 400), nf=0,
                    grid=rng.choice((64, 100, 128)), levels=rng.choice((1, 2)), physics=True,
                    r_obs=robs(60.0, 200.0), dt=-10.0, n_dump=rng.randint(6, 30))
    if kind == "thermal":
        return dict(kind="numerical", precision="mixed", w=_log(rng, 24, 200), h=_log(rng, 24, 160),
                    nf=rng.randint(1, 5), grid=rng.choice((48, 64, 97)), levels=rng.choice((1, 2)),
                    physics=rng.random() < 0.5, r_obs=robs(25.0, 38.0), dt=-2.0, n_dump=rng.randint(2, 6))
    return dict(kind="numerical", precision="fp64", w=_log(rng, 16, 96), h=_log(rng, 16, 72),
                nf=rng.choice((0, 0, 1, 4)), grid=rng.choice((48, 64, 97)), levels=rng.choice((1, 2)),
                physics=rng.random() < 0.5, r_obs=robs(25.0, 38.0), dt=-2.0, n_dump=rng.randint(2, 6))


# ------------------------------------------------------------------ inputs

def _camera(case, rng):
    """One render's parameters: the workload's constants, the seed's camera."""
    c = dict(configs.TORUS_RT_1024, a_spin=rng.uniform(0.0, 0.998), i_obs=rng.uniform(5.0, 85.0),
             j_obs=rng.uniform(0.0, 360.0), n_width=case["w"], n_height=case["h"], r_obs=case["r_obs"],
             n_dump=case["n_dump"], nu=NU_TORUS[:case["nf"]], dt_dump=DT, n_sub=N_SUB,
             precision=api.PREC_FP64 if case.get("precision") == "fp64" else api.PREC_MIXED)
    if case["kind"] == "numerical":
        c.update(configs.NUMERICAL_BASE)
        c.update(i_obs=rng.uniform(5.0, 85.0), j_obs=rng.uniform(0.0, 360.0), n_width=case["w"],
                 n_height=case["h"], r_obs=case["r_obs"], dt_dump=case["dt"], n_dump=case["n_dump"],
                 n_sub=100, nu=NU_THERMAL[:case["nf"]], flow_te=TE, flow_b=B_FIELD)
        if not case["physics"]:
            c.update(w_img=30.0, h_img=30.0)
    return c


def _cameras(case, seed):
    rng = random.Random(seed)
    if case["kind"] == "batch":
        # sides log-uniform between the bounds, the same ones for every seed, smallest first
        n = case["count"]
        sides = [int(round(case["lo"] * (case["hi"] / case["lo"]) ** ((k + 0.5) / n))) for k in range(n)]
        return [_camera(dict(case, w=v, h=v, r_obs=rng.uniform(100.0, 1000.0)), rng) for v in sides]
    return [_camera(case, rng) for _ in range(case.get("count", 1))]


def _times(case):
    """The level times: the workload's (0, 10 M) for rays traced backward
    through flat space, else the pair the trace runs between."""
    if case["levels"] == 1:
        return (0.0, 0.0)
    return (0.0, 10.0) if case["physics"] else (-10.0, 0.0)


def _spacetime(case, seed):
    return dict(a=random.Random(seed + 7).uniform(0.3, 0.9), v=0.3, axis=1)


class State:
    """What the program keeps: context, renders, buffers."""

    def __init__(self):
        self.ctx, self.renders, self.batch, self.out = None, [], None, []

    def __del__(self):
        if self.ctx is not None:
            self.ctx.close()
            self.ctx = None


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def prepare(case, seed):
    s = State()
    s.kind, s.case = case["kind"], case
    cams = _cameras(case, seed)
    if s.kind == "noalloc":
        descs = [api.make_desc(c) for c in cams]
        s.descs = (api.RenderDesc * len(descs))(*descs)
        n, nd = case["w"] * case["h"], 8 + 2 * case["nf"]
        s.out = [(torch.empty((nd, n), dtype=torch.float64, device="cuda"),
                  torch.empty(n, dtype=torch.float64, device="cuda")) for _ in cams]
        s.data = (ctypes.c_void_p * len(cams))(*[d.data_ptr() for d, _ in s.out])
        s.info = (ctypes.c_void_p * len(cams))(*[i.data_ptr() for _, i in s.out])
        return s
    s.ctx = api.Context(0)
    if s.kind == "numerical":
        t1, t2 = _times(case)
        g = api.make_grid(case["grid"], -BOX, BOX, t1, t2, physics=case["physics"])
        bks = _spacetime(case, seed)
        for level, t in enumerate((t1, t2)[:case["levels"]]):
            s.ctx.make_boosted_ks(g, bks["a"], bks["v"], bks["axis"], t, level)
    s.renders = [s.ctx.render(c) for c in cams]
    if s.kind == "batch":
        s.batch = s.ctx.batch(s.renders)
    for r in s.renders:
        if s.kind == "dumps":
            shape = (r.n_data, r.n_rays) if case["layout"] == "soa" else (r.n_rays, r.n_data)
            s.out.append((_pinned(case["n_dump"] + 1, *shape), _pinned(case["n_dump"] + 1, r.n_rays)))
        else:
            s.out.append((_pinned(r.n_data, r.n_rays), _pinned(r.n_rays)))
    return s


# -------------------------------------------------------------------- a pass

def run(s):
    if s.kind == "noalloc":
        st = api.lib().gray_run_mixed_noalloc(0, s.descs, len(s.descs), s.data, s.info,
                                              torch.cuda.current_stream().cuda_stream, None)
        if st != api.OK:
            raise RuntimeError(api.strerror(st))
        return s.out
    if s.kind == "dumps":
        r, (data, info), layout = s.renders[0], s.out[0], LAYOUT[s.case["layout"]]
        d = r.desc
        r.icond()
        r.state(layout, data[0], info[0])
        for i in range(d.n_dump):
            r.evolve(d.t_init + i * d.dt_dump, d.t_init + (i + 1) * d.dt_dump)
            r.state(layout, data[i + 1], info[i + 1])
        return s.out
    if s.batch is not None:
        s.batch.run()
    else:
        s.renders[0].run()
    for r, (data, info) in zip(s.renders, s.out):
        r.state(api.LAYOUT_SOA, data, info)
    return s.out


# ------------------------------------------------------------ work of a pass

def _rays(case):
    if case["kind"] == "batch":
        lo, hi = case["lo"], case["hi"]
        mean = lo * lo if hi == lo else (hi * hi - lo * lo) / (2.0 * math.log(hi / lo))
        return case["count"] * mean
    return case["w"] * case["h"] * case.get("count", 1)


def work(case):
    n, nf = _rays(case), case["nf"]
    state = 8.0 * (8 + 2 * nf) * n + 8.0 * n
    if case["kind"] != "numerical":
        per = flops.fp64_per_step(nf) if case.get("precision") == "fp64" else flops.mixed_per_step(nf)
        reads = case["n_dump"] + 1 if case["kind"] == "dumps" else 1
        return {"bytes": state * reads, "flops": per * float(n) * N_SUB * case["n_dump"]}
    # one contraction of the 8 corners' 40 Gamma per level and stage, where
    # the ray is inside the box; the transfer where there is some
    path = -case["dt"] * case["n_dump"]
    inside = min(1.0, 2.0 * BOX / path) if case["physics"] else 1.0
    used = 1 if case["physics"] else case["levels"]
    per = 4 * (used * (8 * 80 + 72) + 60 + 50 * nf) + 16 * (8 + 2 * nf)
    cells = 160.0 * used * case["grid"] ** 3
    return {"bytes": state + cells, "flops": per * inside * float(n) * path / 0.01}


# --------------------------------------------------- the same in 64 bits

def _intervals(c):
    return c["n_dump"], c["dt_dump"], c["n_sub"]


def _camera_rays(c, dev):
    w, h = c["n_width"], c["n_height"]
    g = torch.arange(w * h, device=dev, dtype=torch.float64)
    gj = torch.floor((g + 0.5) / w)
    gi = g - gj * w
    al = ((gi + 0.5) / w - 0.5) * c["w_img"]
    be = ((gj + 0.5) / h - 0.5) * c["h_img"]
    i, j = math.radians(c["i_obs"]), math.radians(c["j_obs"])
    ci, si, cj, sj = math.cos(i), math.sin(i), math.cos(j), math.sin(j)
    R0 = c["r_obs"] * si - be * ci
    q = torch.stack([torch.zeros_like(g), R0 * cj - al * sj, R0 * sj + al * cj, c["r_obs"] * ci + be * si])
    u = torch.stack([torch.ones_like(g), torch.full_like(g, si * cj), torch.full_like(g, si * sj),
                     torch.full_like(g, ci)])
    return q, u


def _ks(a, q):
    """Kerr-Schild r, f and l_i (covariant, l_t = 1), with r^2 + a^2."""
    x, y, z = q[1], q[2], q[3]
    kk = 0.5 * (x * x + y * y + z * z - a * a)
    rr = kk + torch.sqrt(kk * kk + a * a * z * z)
    r = torch.sqrt(rr)
    f = 2.0 * rr * r / (rr * rr + a * a * z * z)
    ss = rr + a * a
    return r, f, torch.stack([(r * x + a * y) / ss, (r * y - a * x) / ss, z / r]), ss


def _kerr_rhs(c, nu, y):
    """Geodesics from H = g^{mu nu} k_mu k_nu / 2, and the torus transfer."""
    a = c["a_spin"]
    q, kt, k = y[0:4], y[4], y[5:8]
    r, f, l, ss = _ks(a, q)
    x, yy, z = q[1], q[2], q[3]
    rr = r * r
    L = (l * k).sum(0) - kt
    den = r * (rr * rr + a * a * z * z)                     # r^4 + a^2 z^2, times r
    dr = torch.stack([rr * rr * x, rr * rr * yy, rr * ss * z]) / den
    S = rr * rr + a * a * z * z
    df_r = f / r * (3.0 - 4.0 * rr * rr / S)
    dL_r = (x * k[0] + yy * k[1] - 2.0 * r * (l[0] * k[0] + l[1] * k[1])) / ss - z / rr * k[2]
    dL = dL_r * dr + torch.stack([(r * k[0] - a * k[1]) / ss, (a * k[0] + r * k[1]) / ss, k[2] / r])
    df = df_r * dr
    df[2] = df[2] - f * 2.0 * a * a * z / S
    ds = torch.empty_like(y)
    ds[0] = f * L - kt
    ds[1:4] = k - (f * L) * l
    ds[4] = 0.0
    ds[5:8] = f * L * dL + 0.5 * L * L * df
    n = len(nu)
    if n:
        rp = 1.0 + math.sqrt(1.0 - a * a)
        z1 = 1.0 + (1.0 - a * a) ** (1 / 3) * ((1.0 + a) ** (1 / 3) + (1.0 - a) ** (1 / 3))
        z2 = math.sqrt(3.0 * a * a + z1 * z1)
        risco = 3.0 + z2 - math.sqrt((3.0 - z1) * (3.0 + z1 + 2.0 * z2))
        R2 = x * x + yy * yy
        Om = 1.0 / (r * torch.sqrt(r) + a)
        lv = 1.0 - a * Om * R2 / ss
        D = 1.0 - Om * Om * R2 - f * lv * lv
        ut = 1.0 / torch.sqrt(torch.where(D > 0, D, torch.ones_like(D)))
        sh = -ut * (kt + Om * (x * k[1] - yy * k[0]))
        ok = (r > risco) & (D > 0) & (sh > 0)
        sh = torch.where(ok, sh, torch.ones_like(sh))
        h = c["torus_hr"] * r
        dens = torch.where(ok, c["torus_n0"] * (rp / r) ** 1.5 * torch.exp(-z * z / (2.0 * h * h)),
                           torch.zeros_like(r))
        nus = torch.tensor(nu, device=y.device, dtype=torch.float64).unsqueeze(1)
        ds[8:8 + n] = -(dens * sh ** -2.7) * nus ** -0.7 * torch.exp(-y[8 + n:])
        ds[8 + n:] = -(c["torus_kappa"] * dens / sh) / nus ** 2
    return ds


def _rk4(rhs, y, h):
    k1 = rhs(y)
    k2 = rhs(y + 0.5 * h * k1)
    k3 = rhs(y + 0.5 * h * k2)
    k4 = rhs(y + h * k3)
    return y + h / 6.0 * (k1 + 2.0 * (k2 + k3) + k4)


def _exact_kerr(c, dev):
    """The state after every dump interval, the camera's first."""
    nu, a = list(c["nu"]), c["a_spin"]
    n_dump, dt, n_sub = _intervals(c)
    q, u = _camera_rays(c, dev)
    _, f, l, _ = _ks(a, q)
    lu = (l * u[1:]).sum(0)
    A, B, C = f - 1.0, 2.0 * f * lu, (u[1:] ** 2).sum(0) + f * lu * lu
    u[1:] = u[1:] / (-(B + torch.sqrt(B * B - 4.0 * A * C)) / (2.0 * A))

    def lower(q, u):
        _, f, l, _ = _ks(a, q)
        s = f * (u[0] + (l * u[1:]).sum(0))
        return torch.cat([(s - u[0]).unsqueeze(0), u[1:] + s * l])

    def raised(y):
        _, f, l, _ = _ks(a, y[0:4])
        s = f * ((l * y[5:8]).sum(0) - y[4])
        return torch.cat([y[0:4], (s - y[4]).unsqueeze(0), y[5:8] - s * l, y[8:]])

    y = torch.cat([q, lower(q, u), torch.zeros(2 * len(nu), q.shape[1], dtype=torch.float64, device=dev)])
    out = [raised(y)]
    for _ in range(n_dump):  # far from the hole every step is the cap
        for _ in range(n_sub):
            y = _rk4(lambda s: _kerr_rhs(c, nu, s), y, dt / n_sub)
        out.append(raised(y))
    return out


def _boosted_ks(q, a, v, axis):
    """g_{mu nu} of boosted Kerr-Schild at the events q[4, n]."""
    gam = 1.0 / math.sqrt(1.0 - v * v)
    X = list(q)
    X[axis] = gam * (q[axis] - v * q[0])
    x, y, z = X[1], X[2], X[3]
    w = x * x + y * y + z * z - a * a
    r2 = 0.5 * w + torch.sqrt(0.25 * w * w + a * a * z * z)
    r = torch.sqrt(r2)
    ct = z / r
    h = r / (r2 + a * a * ct * ct)
    l = [torch.ones_like(r), (r * x + a * y) / (r2 + a * a), (r * y - a * x) / (r2 + a * a), ct]
    l0, la = l[0], l[axis]
    l[0], l[axis] = gam * (l0 - v * la), gam * (la - v * l0)
    l = torch.stack(l)
    eta = torch.diag(torch.tensor([-1.0, 1.0, 1.0, 1.0], dtype=q.dtype, device=q.device))
    return eta[:, :, None] + 2.0 * h * l[:, None] * l[None, :]


def _nodes(n, dev):
    lo = math.asinh(BOX) ** (1 / 3)
    f = -lo + (2.0 * lo / (n - 1)) * torch.arange(n, dtype=torch.float64, device=dev)
    return torch.sinh(f * f * f)


def _fields(n, t, bks, dev):
    """[n^3, 51] in single precision, as a snapshot file holds them: Gamma^i_jk, g_ij, rho."""
    x = _nodes(n, dev)
    zz, yy, xx = torch.meshgrid(x, x, x, indexing="ij")
    q = torch.stack([torch.full_like(xx, t), xx, yy, zz]).reshape(4, -1)
    fn = lambda p: _boosted_ks(p, bks["a"], bks["v"], bks["axis"])  # noqa: E731
    dg = []
    for w in range(4):
        e = torch.zeros_like(q)
        e[w] = 1.0
        g, d = torch.func.jvp(fn, (q,), (e,))
        dg.append(d)
    dg = torch.stack(dg)                                     # dg[w][i][j] = d_w g_ij
    gu = torch.linalg.inv(g.permute(2, 0, 1)).permute(1, 2, 0)
    low = dg.permute(1, 2, 0, 3) + dg.permute(1, 0, 2, 3) - dg   # [m, b, c]
    cols = []
    for i in range(4):
        for b in range(4):
            for cc in range(b, 4):
                cols.append(0.5 * (gu[i] * low[:, b, cc]).sum(0))
    for i in range(4):
        for j in range(i, 4):
            cols.append(g[i, j])
    cols.append(1.0 / torch.sqrt(q[1] ** 2 + q[2] ** 2 + q[3] ** 2))
    return torch.nan_to_num(torch.stack(cols, 1), posinf=float("inf"), neginf=float("-inf")).float().double()


def _interp(levels, times, n, physics, q):
    """All 51 fields at the events: trilinear in the logical coordinates, linear in time."""
    x = _nodes(n, q.device)
    i0, w = [], []
    for a in range(3):
        p = q[a + 1].contiguous()
        i = (torch.searchsorted(x, p, right=True) - 1).clamp(0, n - 2)
        f = ((p - x[i]) / (x[i + 1] - x[i])).clamp(0.0, 1.0)
        i0.append(i)
        w.append(f)
    bits = torch.arange(8, device=q.device)
    c = [(bits >> a) & 1 for a in range(3)]                 # the eight corners' x, y and z sides
    ia = [i0[a] + c[a].unsqueeze(1) for a in range(3)]
    wa = [torch.where(c[a].unsqueeze(1) == 1, w[a], 1 - w[a]) for a in range(3)]
    row, wt = (ia[2] * n + ia[1]) * n + ia[0], (wa[0] * wa[1] * wa[2]).unsqueeze(2)
    v = [(wt * f[row]).sum(0) for f in levels]
    if len(levels) == 1:
        return v[0].t()
    ft = (q[0] - times[0]) / (times[1] - times[0])
    if physics:
        ft = ft.clamp(0.0, 1.0)
    return (v[0] + ft.unsqueeze(1) * (v[1] - v[0])).t()


def _thermal(c, nu, k, ne, tau):
    """dI/dl and dtau/dl [nf, n] of thermal bremsstrahlung and synchrotron in CGS."""
    cl, hp, G, Ry, e, me, msun, kb = (2.99792458e10, 6.62606957e-27, 6.673848e-8, 2.17987197e-11,
                                      4.80320425e-10, 9.10938291e-28, 1.9891e33, 1.38064881e-16)
    te, b, eps, m = c["flow_te"], c["flow_b"], 1e-28, api.DEFAULTS["m_adm"]
    sh = -k[0]
    cos = k[3] * b / (sh * b + eps)
    v = nu * sh
    f2 = hp / (me * cl) * (v / cl) / te
    B = torch.where(f2 > 1e-5, 2 * hp * v ** 3 / cl ** 2 / torch.expm1(f2.clamp(min=1e-5)),
                    2 * hp * v ** 3 / cl ** 2 / f2 / (1 + f2 / 2 + f2 * f2 / 6))
    y = hp / (me * cl * cl) * v / te                        # te >> 1: the hot branches of the Gaunt factor
    gaunt = torch.where(y > 1, math.sqrt(3 / math.pi) / torch.sqrt(y),
                        math.sqrt(3) / math.pi * (math.log(4 / 1.78107241799) - torch.log(y + eps)))
    ff = G * msun / (cl * cl) * 6.8e-38 / (4 * math.pi * math.sqrt(me * cl * cl / kb))
    Lff = m * ff * ne * ne * gaunt / (math.sqrt(te) * torch.exp(y) + eps)
    nus = te * te * b * torch.sqrt((1 - cos * cos).clamp(min=0.0)) * (e / (9 * math.pi * me * cl))
    xs = v / (nus + eps)
    xx = torch.sqrt(xs) + 1.88774862536 * xs ** (1 / 6)
    Ls = m * xx * xx * torch.exp(-xs ** (1 / 3)) / (2 * te * te - 0.5) * ne * nus * \
        (G * msun / cl ** 2) * (math.sqrt(2) * math.pi * e * e / (3 * cl))
    L = Lff + torch.where((cos > -1) & (cos < 1), Ls, torch.zeros_like(Ls))
    return -L * torch.exp(-tau) / (sh * sh), -L * sh / (B + eps)


def _exact_numerical(case, c, seed, dev):
    nu = list(c["nu"])
    times = _times(case)
    levels = [_fields(case["grid"], t, _spacetime(case, seed), dev) for t in times[:case["levels"]]]
    idx = {}
    n = 0
    for i in range(4):
        for j in range(i, 4):
            idx[i, j] = idx[j, i] = n
            n += 1

    def fields(q):
        v = _interp(levels, times, case["grid"], case["physics"], q)
        if case["physics"]:
            out = ~((q[1:4].abs() <= BOX).all(0))
            flat = torch.zeros(51, 1, dtype=v.dtype, device=v.device)
            flat[40 + idx[0, 0]] = -1.0
            for i in (1, 2, 3):
                flat[40 + idx[i, i]] = 1.0
            v = torch.where(out, flat, v)
        return v

    def lowered(v, u):
        return torch.stack([sum(v[40 + idx[i, j]] * u[j] for j in range(4)) for i in range(4)])

    def rhs(s):
        q, u = s[0:4], s[4:8]
        v = fields(q)
        p = torch.stack([u[i] * u[j] * (1.0 if i == j else 2.0) for i in range(4) for j in range(i, 4)])
        g = [(v[10 * m:10 * m + 10] * p).sum(0) for m in range(4)]
        ds = torch.empty_like(s)
        ds[0:4] = u
        for m in range(4):
            ds[4 + m] = g[0] * u[m] - g[m]
        if nu:
            k = lowered(v, u)
            ds[8:8 + len(nu)], ds[8 + len(nu):] = _thermal(c, nus, k, v[50], s[8 + len(nu):])
        return ds

    nus = torch.tensor(nu, dtype=torch.float64, device=dev).unsqueeze(1)
    q, u = _camera_rays(c, dev)
    s = torch.cat([q, u, torch.zeros(2 * len(nu), q.shape[1], dtype=torch.float64, device=dev)])
    n_dump, dt, n_sub = _intervals(c)
    steps = int(round(n_dump * -dt / 0.01))
    for _ in range(steps):
        s = _rk4(rhs, s, -0.01)
    return s, (lowered(fields(s[0:4]), s[4:8]) * s[4:8]).sum(0)


def exact(case, seed):
    """Where every step is the cap and no ray comes near the horizon; a whole
    path through the hole's region takes minutes in this form."""
    cams = _cameras(case, seed)
    dev = "cuda"
    if case["kind"] == "numerical":
        path = -case["dt"] * case["n_dump"]
        if path > 12.0 or case["r_obs"] - path < 13.0 or case["physics"] and case["r_obs"] > BOX:
            return None
        s, info = _exact_numerical(case, cams[0], seed, dev)
        return [(s, info)]
    path = -DT * case["n_dump"]
    if case["kind"] == "batch" or min(c["r_obs"] for c in cams) - path < 6.0 or len(cams) * path > 100.0:
        return None
    # g(u, u) of a null ray is 0 and what comes back for it is rounding: no value
    runs = [_exact_kerr(c, dev) for c in cams]
    if case["kind"] != "dumps":
        return [(r[-1], None) for r in runs]
    swap = (lambda t: t.t()) if case["layout"] == "aos" else (lambda t: t)
    return [(torch.stack([swap(s) for s in r]), None) for r in runs]
