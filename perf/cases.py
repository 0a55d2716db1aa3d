"""Measured cases of the framework: the calls a simulation program makes, over its range of sizes.

A program that uses thorx builds a grid and a context, sets the state, and then repeats the large
step (ProfX + Thor as one graph replay, thorx_step), with or without the double-gray RT and the
Rayleigh sponge, in the all-FP64 or the mixed form; a host program that keeps its own loop calls
thorx_profx and thorx_thor itself, or takes the state in and out every step; between steps it sums
the global diagnostics, and with the RT surrogate it trains the network. Each listed case is one of
these calls; draw() gives others of the same ranges.

The initial state is the configurations' own (isothermal 300 K or the Guillot profile, in the
model's discrete hydrostatic balance, with seeded temperature noise) plus a zonal wind with seeded
noise and a small vertical momentum, so that every term of the step is at work.

exact() is a plain torch restatement of the step in 64 bits (finite-volume sums written out, no
operator weights, no code of this repository; the grid arrays, which are inputs, are the same).
"""
import math

import numpy as np
import torch

import thor_b200

DEV = "cuda"
EARTH = dict(A=6.371e6, Omega=7.292e-5, Gravit=9.8, Rd=287.0, Cp=1005.0, P_Ref=1e5,
             Top_altitude=36e3, Diffc=0.0048, DivDampc=0.0048, HyDiffOrder=4, DeepModel=1,
             NonHydro=1, GravHeightVar=0, HyDiff=1, DivDampP=1, thermo_equation=0,
             core_benchmark=1, precision=0)
# the hot Jupiter of the RT configuration: T_irr 2000 K, 100 bar at the bottom, 1e-3 bar at the top
HJ_TEQ = 2000.0 / 2 ** 0.5
HOT_JUPITER = dict(EARTH, A=1e8, Omega=9.09e-5, Gravit=10.0, Rd=3714.0, Cp=13000.0, P_Ref=1e7,
                   Top_altitude=3714.0 * HJ_TEQ / 10.0 * math.log(1e7 / 1e2), Diffc=0.015,
                   DivDampc=0.015, core_benchmark=0)
RT_HJ = dict(Tstar=4300.0, radius_star=0.667 * 695700000.0,
             planet_star_dist=0.667 * 695700000.0 * (4300.0 / 2000.0) ** 2, diff_ang=0.5,
             Tint=100.0, albedo=0.0, kappa_sw=4e-4, kappa_lw=1e-3, kappa_lw_pole=1e-3, n_sw=1.0,
             n_lw=2.0, f_lw=0.5, sync_rot=1, alpha_i=0.0)
RT_EARTH = dict(Tstar=5772.0, radius_star=695700000.0, planet_star_dist=149597870700.0,
                diff_ang=0.5, Tint=0.0, albedo=0.3, kappa_sw=4e-4, kappa_lw=1e-3,
                kappa_lw_pole=1e-3, n_sw=1.0, n_lw=2.0, f_lw=0.5, sync_rot=0,
                mean_motion=1.991e-7, alpha_i=0.0)
SPONGE_BINS = 20
STATE_OUT = ["Rho", "pressure", "Mh", "Wh", "W", "temperature"]
STATE_IO = ["Rho", "pressure", "Mh", "Wh"]
RT_OUT = ["flw_up", "flw_dn", "fsw_dn", "tau", "insol", "ASR", "OLR"]
BATCH, HIDDEN, ADAM_STEPS, ADAM_LR = 8192, 512, 20, 1e-3


def _case(name, call, glevel, nv, planet="earth", mixed=False, rt=False, sponge=False, deep=True,
          nonhydro=True, energy=False, varying=False):
    c = dict(call=call, glevel=glevel, nv=nv, planet=planet, mixed=mixed, rt=rt, sponge=sponge,
             deep=deep, nonhydro=nonhydro, energy=energy, varying=varying)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # Held-Suarez at the smallest resolution in use: what launches and latency cost
        _case("step_hs_g4_L32", "step", 4, 32),
        # the quasi-hydrostatic shallow model with the energy equation, an odd number of levels
        _case("step_shallow_energy_g5_L37", "step", 5, 37, deep=False, nonhydro=False, energy=True),
        # the hot Jupiter with double-gray RT
        _case("step_hj_rt_g5_L40", "step", 5, 40, planet="hj", rt=True),
        # the same with the Rayleigh sponge at the top, in the mixed form
        _case("step_hj_rt_sponge_mixed_g5_L40", "step", 5, 40, planet="hj", rt=True, sponge=True,
              mixed=True),
        # the headline workload in both forms
        _case("step_hs_g6_L48", "step", 6, 48),
        _case("step_hs_mixed_g6_L48", "step", 6, 48, mixed=True),
        # the large run: Held-Suarez with RT, mixed, all state resident
        _case("step_hs_rt_mixed_g7_L48", "step", 7, 48, rt=True, mixed=True),
        # the dynamical core called by a host program's own loop, Rd and Cp varying by cell
        _case("thor_varying_g6_L33", "thor", 6, 33, varying=True),
        # the physics pass called by a host program's own loop
        _case("profx_hj_rt_g6_L48", "profx", 6, 48, planet="hj", rt=True),
        # state in from and out to pinned host memory around each step (a host program that keeps
        # its own arrays, or writes every step)
        _case("exchange_hs_g6_L48", "exchange", 6, 48),
        # the conservation diagnostics
        _case("globdiag_g6_L48", "globdiag", 6, 48),
        # Adam steps of the RT surrogate on a batch of 8192 logged columns
        _case("train_g5_L40", "train", 5, 40, planet="hj", rt=True),
    ]


def draw(rng):
    call = rng.choice(["step"] * 6 + ["thor", "profx", "exchange", "globdiag"])
    glevel = rng.choice([4, 5, 5, 6, 6])
    nv = int(round(math.exp(rng.uniform(math.log(12), math.log(64)))))
    planet = rng.choice(["earth", "earth", "hj"])
    deep = rng.random() < 0.8
    return _case(None, call, glevel, nv, planet=planet, mixed=rng.random() < 0.4,
                 rt=call in ("step", "profx") and (planet == "hj" or rng.random() < 0.2),
                 sponge=call in ("step", "profx") and rng.random() < 0.25, deep=deep,
                 nonhydro=rng.random() < 0.75, energy=rng.random() < 0.25,
                 varying=rng.random() < 0.2)


# ---- inputs -------------------------------------------------------------------------------------
_grids = {}


def _grid(case):
    p = _planet(case)
    key = (case["glevel"], case["nv"], case["planet"])
    if key not in _grids:
        # spring dynamics where it takes no longer than the rest of the set-up
        _grids[key] = thor_b200.Icogrid(case["glevel"], case["nv"], A=p["A"],
                                        Top_altitude=p["Top_altitude"],
                                        spring=case["glevel"] <= 5).as_dict()
    return _grids[key]


def _planet(case):
    return dict(EARTH if case["planet"] == "earth" else HOT_JUPITER)


def _timestep(case):
    if case["planet"] == "hj":
        return 600.0 if case["glevel"] <= 4 else 300.0 if case["glevel"] == 5 else 150.0
    return 1200.0 * 2.0 ** (4 - case["glevel"])


def _rt(case):
    return dict(RT_EARTH if case["planet"] == "earth" else RT_HJ)


def _params(case):
    p = _planet(case)
    p.update(timestep=_timestep(case), precision=int(case["mixed"]), DeepModel=int(case["deep"]),
             NonHydro=int(case["nonhydro"]), thermo_equation=int(case["energy"]))
    return p


def _guillot(p, c, rt):
    mu, kl, ks, f = 0.5, rt["kappa_lw"], rt["kappa_sw"], rt["f_lw"]
    eps, x0, g0 = 1.0 / f, c["P_Ref"] / c["Gravit"], ks / kl
    tau0 = kl * x0
    tau, s = kl * p / c["Gravit"], p / c["P_Ref"]
    gam = ks / (kl * (1.0 + 2 * (eps - 1) * s))
    e = math.exp(-g0 * tau / mu)
    t4 = (0.75 * rt["Tint"] ** 4 * (2. / 3 + tau0 * s + (eps - 1) * tau0 * s * s)
          + 3 * mu * HJ_TEQ ** 4 * (2. / 3 + gam / (3 * mu) * e + mu / g0 * (1.0 - e)
                                    + 2 * (eps - 1) * mu / (g0 * ks * x0)
                                    * (mu - (mu + g0 * tau) * e)))
    return t4 ** 0.25


def _column(case, alt, alth):
    """(p, T) of the rest column in the model's discrete hydrostatic balance."""
    c, rt = _planet(case), _rt(case)
    temp = (lambda p: 300.0) if case["planet"] == "earth" else (lambda p: _guillot(p, c, rt))
    nv, g, Rd = len(alt), c["Gravit"], c["Rd"]
    p, T = np.zeros(nv), np.zeros(nv)
    for l in range(nv):
        if l == 0:
            pl, Tl, dz, a, b = c["P_Ref"], temp(c["P_Ref"]), alt[0], 0.5, 0.5
        else:
            pl, Tl, dz = p[l - 1], T[l - 1], alt[l] - alt[l - 1]
            a, b = (alt[l] - alth[l]) / dz, (alth[l] - alt[l - 1]) / dz
        p[l], T[l] = pl, Tl
        for _ in range(200):
            f = (p[l] - pl) / dz + g * (p[l] * b / (Rd * T[l]) + pl * a / (Rd * Tl))
            d = f / (1.0 / dz + g * b / (Rd * T[l]))
            p[l] -= d
            T[l] = temp(p[l])
            if abs(d) <= 1e-15 * p[l]:
                break
    return p, T


def _inputs(case, seed):
    """The initial state in the reference layouts ([col][lev], [col][lev][xyz], [col][lev+1])."""
    g, c = _grid(case), _planet(case)
    N, nv = g["point_num"], case["nv"]
    rng = np.random.Generator(np.random.PCG64(seed))
    alt, alth = np.asarray(g["Altitude"]), np.asarray(g["Altitudeh"])
    p0, T0 = _column(case, alt, alth)
    hj = case["planet"] == "hj"
    T = T0[None, :] + (1.0 if hj else 0.1) * (2.0 * rng.random((N, nv)) - 1.0)
    p = np.broadcast_to(p0, (N, nv)).copy()
    ones = np.ones((N, nv))
    Rd, Cp = c["Rd"] * ones, c["Cp"] * ones
    if case["varying"]:
        Rd *= 1.0 + 0.002 * (2.0 * rng.random((N, nv)) - 1.0)
        Cp *= 1.0 + 0.002 * (2.0 * rng.random((N, nv)) - 1.0)
    rho = p / (Rd * T)
    lon, lat = np.asarray(g["lonlat"])[0::2], np.asarray(g["lonlat"])[1::2]
    U = 100.0 if hj else 10.0
    u = (U * np.cos(lat) ** 2)[:, None] * np.sin(np.pi * alt / alth[-1])[None, :]
    u = u + 0.02 * U * (2.0 * rng.random((N, nv)) - 1.0)
    v = 0.02 * U * (2.0 * rng.random((N, nv)) - 1.0)
    east = np.stack([-np.sin(lon), np.cos(lon), 0 * lon], 1)
    north = np.stack([-np.sin(lat) * np.cos(lon), -np.sin(lat) * np.sin(lon), np.cos(lat)], 1)
    Mh = rho[:, :, None] * (u[:, :, None] * east[:, None, :] + v[:, :, None] * north[:, None, :])
    Wh = np.zeros((N, nv + 1))
    Wh[:, 1:nv] = 1e-3 * rho[:, 1:] * (2.0 * rng.random((N, nv - 1)) - 1.0)
    return dict(Rho=rho, pressure=p, temperature=T, Mh=Mh, Wh=Wh, W=np.zeros((N, nv)), Rd=Rd, Cp=Cp)


def _layers(case, seed):
    """Glorot-uniform weights and zero biases of the surrogate, in its padded shapes."""
    nv, rng = case["nv"], np.random.Generator(np.random.PCG64(seed + 77))
    n_in = 2 * nv + 1
    kin, nout = -(-n_in // 64) * 64, -(-nv // 64) * 64
    out = []
    for n, k, nn, kk in ((HIDDEN, kin, HIDDEN, n_in), (HIDDEN, HIDDEN, HIDDEN, HIDDEN),
                         (HIDDEN, HIDDEN, HIDDEN, HIDDEN), (nout, HIDDEN, nv, HIDDEN)):
        W = np.zeros((n, k), np.float32)
        a = math.sqrt(6.0 / (nn + kk))
        W[:nn, :kk] = a * (2.0 * rng.random((nn, kk)) - 1.0)
        out.append((W, np.zeros(n, np.float32)))
    return out


class _Planes:
    """A context's device array [components x levels][plane] for torch.as_tensor; the tensor keeps
    this object, and with it the context that owns the memory."""

    def __init__(self, x, name):
        self.x = x
        ptr, levels, comps, plane = x.device_field(name)
        self.__cuda_array_interface__ = dict(shape=(comps * levels, plane), typestr="<f8",
                                             data=(ptr, False), strides=None, version=3)


def _view(x, name):
    return torch.as_tensor(_Planes(x, name), device=DEV)[:, :x.N]


_stream = []


def _the_stream():
    """One stream for every context, as a program with one simulation has: passes run in turn."""
    if not _stream:
        _stream.append(torch.cuda.Stream())
    return _stream[0]


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.call, s.case = case["call"], case
    s.x = x = thor_b200.Thorx(_grid(case), case["glevel"], _params(case),
                              stream=_the_stream().cuda_stream)
    ic = _inputs(case, seed)
    for k, v in ic.items():
        x.set(k, v)
    if case["rt"]:
        x.rt_enable(_rt(case))
    if case["sponge"]:
        x.sponge(dict(nlat_bins=SPONGE_BINS))
    if s.call in ("step", "thor"):
        s.out = {f: _view(x, f) for f in STATE_OUT}
    elif s.call == "profx":
        s.out = {f: _view(x, f) for f in ["pressure", "Mh", "W", "temperature", "profx_Qheat"]
                 + (RT_OUT if case["rt"] else [])}
    elif s.call == "exchange":
        pin = lambda n: torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()  # noqa: E731
        s.host = {f: pin(x.size(f)) for f in STATE_IO}
        s.back = {f: pin(x.size(f)) for f in STATE_IO}
        for f in STATE_IO:
            s.host[f][:] = ic[f].reshape(-1)
    elif s.call == "train":
        x.sur_create(hidden=HIDDEN, train_batch=BATCH, log_capacity=2 * x.N, seed=1 + seed)
        for l, (W, b) in enumerate(_layers(case, seed)):
            x.sur_set_layer(l, W, b)
        x.sur_mode(thor_b200.SUR_LOG)
        x.profx()
    return s


def run(s):
    x = s.x
    if s.call == "step":
        x.step(1)
        return s.out
    if s.call == "thor":
        x.thor()
        return s.out
    if s.call == "profx":
        x.profx()
        return s.out
    if s.call == "exchange":
        for f in STATE_IO:
            x.set(f, s.host[f])
        x.step(1)
        for f in STATE_IO:
            x.get(f, s.back[f])
        return s.back
    if s.call == "globdiag":
        d = x.globdiag()
        return dict(energy=d[0], mass=d[1], am=np.array(d[2:5]), entropy=d[5])
    losses = x.sur_train(ADAM_STEPS, BATCH, ADAM_LR)
    return [list(x.sur_layer(l)) for l in range(4)] + [np.array(losses)]


def work(case):
    N, nv = 2 + 10 * 4 ** case["glevel"], case["nv"]
    cells = float(N) * nv
    S = 8.0 * cells
    geo = N * 8.0 * (42 + 78) + N * 6 * 4.0  # div, grad, ring geometry, neighbours
    call = case["call"]
    rt_bytes = S * 7.0 if case["rt"] else 0.0  # heating, two opacities, four flux profiles
    rt_flops = cells * 250.0 if case["rt"] else 0.0
    # operations a cell needs in a large step: 3 stages x (advection and thermodynamics 350, two
    # Laplacians of six variables 250, divergence damping 350, slow modes 250) and 10 small steps
    # x (divergence damping 350, momentum 100, vertical solve and update 350)
    thor = cells * (3 * 1200.0 + 10 * 800.0)
    profx = cells * 120.0
    if call == "step":
        return dict(bytes=6 * S + 8 * S + geo + rt_bytes, flops=thor + profx + rt_flops)
    if call == "thor":
        return dict(bytes=(7 + (2 if case["varying"] else 0)) * S + 8 * S + geo, flops=thor)
    if call == "profx":
        return dict(bytes=6 * S + 7 * S + rt_bytes, flops=profx + rt_flops)
    if call == "exchange":
        return dict(bytes=2 * 6 * S + 14 * S + geo, flops=thor + profx)
    if call == "globdiag":
        return dict(bytes=9 * S, flops=cells * 80.0)
    n_in, kin, nout = 2 * nv + 1, -(-(2 * nv + 1) // 64) * 64, -(-nv // 64) * 64
    weights = kin * HIDDEN + 2 * HIDDEN * HIDDEN + HIDDEN * nout
    return dict(bytes=ADAM_STEPS * (4.0 * BATCH * (n_in + nv) + 4.0 * 7 * weights),
                flops=ADAM_STEPS * 6.0 * BATCH * weights)


def tolerance(case):
    """About four times the largest error against exact() seen over the ranges after two passes."""
    if case["call"] == "globdiag":
        return dict(rel=2e-14)
    if case["call"] == "train":  # bf16 gradients: Adam's step of a weight with a small one flips sign
        return dict(rel=2e-2)
    if case["call"] == "profx":
        return dict(rel=1e-13)
    # the vertical momentum, a small residual of the hydrostatic balance, carries the largest error
    return dict(rel=5e-8 if case["mixed"] else 2e-10)


# ---- the step in plain torch, 64 bits -----------------------------------------------------------
class _Exact:
    def __init__(self, case, ic):
        g, p = _grid(case), _params(case)
        self.case, self.p = case, p
        self.N, self.nv = N, nv = g["point_num"], case["nv"]
        f = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=DEV)  # noqa: E731
        self.alt, self.alth = f(g["Altitude"])[:, None], f(g["Altitudeh"])[:, None]
        self.lon, self.lat = f(np.asarray(g["lonlat"])[0::2]), f(np.asarray(g["lonlat"])[1::2])
        self.areasT = f(g["areasT"])[:N]
        geo = lambda k, *sh: f(np.asarray(g[k]).reshape((N,) + sh)).movedim(0, -1)  # noqa: E731
        self.AR, self.AT = geo("areas", 6, 3), geo("areasTr", 6)
        self.TI, self.TE, self.OA = geo("nvecti", 6, 3), geo("nvecte", 6, 3), geo("nvecoa", 6, 3)
        self.div, self.grad = geo("div", 7, 3), geo("grad", 7, 3)
        self.fr = geo("func_r", 3)
        self._neighbours(g)
        cell = lambda k: f(ic[k].reshape(N, nv)).t().contiguous()  # noqa: E731
        self.Rho, self.pr, self.T, self.W = (cell(k) for k in ("Rho", "pressure", "temperature", "W"))
        self.Rd, self.Cp = cell("Rd"), cell("Cp")
        self.Mh = f(ic["Mh"].reshape(N, nv, 3)).permute(2, 1, 0).contiguous()
        self.Wh = f(ic["Wh"].reshape(N, nv + 1)).t().contiguous()
        self.Qheat = torch.zeros_like(self.Rho)
        self.steps = 0
        A, alt, alth = p["A"], self.alt, self.alth
        one = torch.ones_like(alt)
        deep = case["deep"]
        self.rs = A / (alt + A) if deep else one
        self.r2c = (alt + A) ** 2 if deep else one
        self.r2h = (alth + A) ** 2 if deep else torch.ones_like(alth)
        self.dz = alth[1:] - alth[:-1]
        self.dr2dz = ((alth[1:] + A) ** 3 - (alth[:-1] + A) ** 3) / 3 if deep else self.dz
        # weights at an interior interface i = 1..nv-1 of the layers below and above
        self.hb = (alth[1:-1] - alt[1:]) / (alt[:-1] - alt[1:])
        self.ha = (alth[1:-1] - alt[:-1]) / (alt[1:] - alt[:-1])
        # weights at a centre of the interfaces below and above
        self.cb = (alt - alth[1:]) / (alth[:-1] - alth[1:])
        self.ca = (alt - alth[:-1]) / (alth[1:] - alth[:-1])
        dbar = math.sqrt(2 * math.pi / 5) * A / 2 ** case["glevel"]
        self.kdh = p["Diffc"] * dbar ** p["HyDiffOrder"] / p["timestep"]
        self.kdz = p["DivDampc"] * dbar ** 4 / p["timestep"]

    def _neighbours(self, g):
        N, nl = self.N, int(g["nl_region"])
        m = np.asarray(g["maps"]).reshape(int(g["nr"]), nl + 2, nl + 2)
        ids = m[:, 1:-1, 1:-1].reshape(-1)
        pts = [m[:, 2:, 1:-1], m[:, 2:, 2:], m[:, 1:-1, 2:], m[:, :-2, 1:-1], m[:, :-2, :-2],
               m[:, 1:-1, :-2]]
        pts = [q.reshape(-1).copy() for q in pts]
        pent = np.zeros(m[:, 1:-1, 1:-1].shape, bool)
        pent[:, 0, 0] = m[:, 0, 0] == -1
        pent = pent.reshape(-1)
        pts[4][pent] = pts[5][pent]
        nb = np.full((6, N), -1, np.int64)
        ring = np.full((6, N), -1, np.int64)
        for j in range(6):
            nb[j, ids] = pts[j]
            ring[j, ids] = np.where(pent & (j == 5), -1, pts[j])
        loc = np.asarray(g["point_local"]).reshape(N, 6)
        for c in (N - 2, N - 1):
            nb[:5, c] = ring[:5, c] = loc[c, :5]
        nb[nb < 0] = N  # a hole: the zero column
        t = lambda a: torch.as_tensor(a, device=DEV)  # noqa: E731
        self.nb = t(nb)
        five = ring[5] < 0
        ring[ring < 0] = N
        self.ring = t(ring)
        self.pole = torch.zeros(N, dtype=torch.bool, device=DEV)
        self.pole[N - 2:] = True
        self.sets = ((t(np.nonzero(~five)[0]), 6), (t(np.nonzero(five)[0]), 5))

    def at(self, a, idx):
        """a at the columns idx, 0 at a hole."""
        return torch.cat([a, torch.zeros_like(a[..., :1])], -1)[..., idx]

    def stencil(self, w, vec):
        """sum over the 7 points and components of w[j][k] vec[k](point j)."""
        out = 0
        for j in range(7):
            v = vec if j == 0 else self.at(vec, self.nb[j - 1])
            for k in range(3):
                out = out + w[j, k] * v[k]
        return out

    def gradient(self, a):
        out = [0, 0, 0]
        for j in range(7):
            v = a if j == 0 else self.at(a, self.nb[j - 1])
            for k in range(3):
                out[k] = out[k] + self.grad[j, k] * v
        return torch.stack([self.rs * o for o in out])

    def laplacian(self, a):
        out = torch.empty_like(a)
        for cols, n in self.sets:
            AR, AT, TI, TE, OA = (q[..., cols] for q in (self.AR, self.AT, self.TI, self.TE, self.OA))
            a0 = a[:, cols]
            p = [self.at(a, self.ring[j][cols]) for j in range(n)]
            gr = []
            for j in range(n):
                q = (j + 1) % n
                m = (AR[j, 0] * a0 + AR[j, 1] * p[j] + AR[j, 2] * p[q]) / AT[j]
                l1, l2, l3 = 0.5 * (p[j] + a0) - m, 0.5 * (p[j] + p[q]) - m, 0.5 * (a0 + p[q]) - m
                gr.append([(-l1 * TI[j, k] + l2 * TE[j, k] + l3 * TI[q, k]) * self.rs / AT[j]
                           for k in range(3)])
            tot = 0
            for j in range(n):
                q = (j + 1) % n
                for k in range(3):
                    tot = tot + (gr[j][k] + gr[q][k]) * OA[j, k] * (0.5 * self.rs)
            out[:, cols] = tot
        return out

    def graddiv(self, M, W=None):
        """The gradient of the divergence (of M and the vertical momentum W at the interfaces)."""
        out = torch.empty_like(M)
        for cols, n in self.sets:
            AR, AT, TI, TE, OA = (q[..., cols] for q in (self.AR, self.AT, self.TI, self.TE, self.OA))
            a0 = M[..., cols]
            p = [self.at(M, self.ring[j][cols]) for j in range(n)]
            if W is not None:
                dw = (W[:-1] - W[1:]) / -self.dz
                w0 = dw[:, cols]
                wp = [self.at(dw, self.ring[j][cols]) for j in range(n)]
            D = []
            for j in range(n):
                q = (j + 1) % n
                d = 0
                for k in range(3):
                    d = d + (-(a0[k] + p[j][k]) * TI[j, k] + (p[j][k] + p[q][k]) * TE[j, k]
                             + (a0[k] + p[q][k]) * TI[q, k])
                d = d * (0.5 * self.rs / AT[j])
                if W is not None:  # the poles weigh the third corner by the second sub-area
                    a2 = torch.where(self.pole[cols], AR[j, 1], AR[j, 2])
                    d = d + (AR[j, 0] * w0 + AR[j, 1] * wp[j] + a2 * wp[q]) / AT[j]
                D.append(d)
            for k in range(3):
                out[k][:, cols] = sum((D[j] + D[(j + 1) % n]) * OA[j, k] * (0.5 * self.rs)
                                      for j in range(n))
        return out

    def tangent(self, M):
        r = (M * self.fr[:, None]).sum(0)
        return M - self.fr[:, None] * r

    def up(self, a):
        """a cell field at the interior interfaces."""
        return a[:-1] * self.hb + a[1:] * self.ha

    def pad(self, a):
        z = torch.zeros_like(a[:1])
        return torch.cat([z, a, z])

    # -- ProfX --
    def profx(self):
        p, alt, nv = self.p, self.alt, self.nv
        self.Qheat = torch.zeros_like(self.Rho)
        self.steps += 1
        dt = p["timestep"]
        self.W = self.Wh[:-1] * self.cb + self.Wh[1:] * self.ca
        if self.case["sponge"]:
            self.sponge()
        self.T = self.pr / (self.Rd * self.Rho)
        if p["core_benchmark"] == 1:
            ps = 0.5 * (self.pr[0] + self.pr[1] - self.Rho[0] * p["Gravit"] * (-alt[0] - alt[1]))
            sg, s0, kappa = self.pr / ps, self.pr / 1e5, p["Rd"] / p["Cp"]
            teq = (315.0 - 60.0 * torch.sin(self.lat) ** 2
                   - 10.0 * torch.log(s0) * torch.cos(self.lat) ** 2) * s0 ** kappa
            teq = teq.clamp(min=200.0)
            b = ((sg - 0.7) / 0.3).clamp(min=0.0)
            ka, ks, kf = 1 / 40.0 / 86400.0, 1 / 4.0 / 86400.0, 1 / 86400.0
            kt = ka + (ks - ka) * b * torch.cos(self.lat) ** 4
            self.Mh = self.Mh / (1.0 + kf * b * dt)
            self.T = self.T - kt * dt * (self.T - teq)
        if self.case["rt"]:
            self.rt()
        self.pr = self.T * self.Rd * self.Rho

    def sponge(self):
        n, dt = SPONGE_BINS, self.p["timestep"]
        lat, lon = self.lat, torch.where(self.lon < 0, self.lon + 2 * math.pi, self.lon)
        d = math.pi / n
        edges = torch.cumsum(torch.tensor([-math.pi / 2] + [d] * n, dtype=torch.float64), 0).to(DEV)
        b = (torch.searchsorted(edges, lat, right=True) - 1).clamp(0, n - 1)
        sl, cl, sp, cp = torch.sin(lon), torch.cos(lon), torch.sin(lat), torch.cos(lat)
        east = torch.stack([-sl, cl, 0 * sl])[:, None]
        north = torch.stack([-sp * cl, -sp * sl, cp])[:, None]
        wind = [(self.Mh * east).sum(0) / self.Rho, (self.Mh * north).sum(0) / self.Rho,
                self.W / self.Rho]
        cnt = torch.zeros(n, dtype=torch.float64, device=DEV).index_add(0, b, torch.ones_like(lat))
        x = (lat + math.pi / 2) / d - 0.5  # bin-centre coordinate
        lo = torch.floor(x).clamp(0, n - 1).long()
        hi = (lo + 1).clamp(max=n - 1)
        fr = torch.where((x < 0) | (x > n - 1), torch.zeros_like(x), x - lo)
        z = self.alt / self.alth[-1]
        s = torch.where(z >= 0.75, torch.sin(0.5 * math.pi * (z - 0.75) / 0.25) ** 2, 0 * z)
        new = []
        for a in wind:
            mean = torch.zeros((self.nv, n), dtype=torch.float64, device=DEV).index_add(1, b, a) / cnt
            m = mean[:, lo] * (1 - fr) + mean[:, hi] * fr
            new.append((a / dt + 1e-4 * s * m) / (1.0 / dt + 1e-4 * s))
        self.Mh = (new[0] * east + new[1] * north) * self.Rho
        self.W = new[2] * self.Rho
        self.Wh = torch.cat([self.Wh[:1], self.up(self.W), self.Wh[-1:]])

    def rt(self):
        r, p, nv, alt, alth = _rt(self.case), self.p, self.nv, self.alt, self.alth
        dt, g = p["timestep"], p["Gravit"]
        n = self.steps
        flux = (r["radius_star"] / r["planet_star_dist"]) ** 2 * 5.6703744191844314e-08 * r["Tstar"] ** 4
        if r["sync_rot"]:
            cz = torch.cos(self.lat) * torch.cos(self.lon)
        else:  # circular orbit without obliquity: true longitude = mean motion x time
            a = -p["Omega"] * n * dt + math.fmod(math.fmod(r["mean_motion"] * n * dt, 2 * math.pi),
                                                 2 * math.pi)
            cz = torch.cos(self.lat) * torch.cos(self.lon - a)
        cz = cz.clamp(min=0.0)
        insol = torch.where(cz > 0, flux * cz, 0 * cz)
        P, T, rho = self.pr, self.T, self.Rho
        ps = 0.5 * (P[0] + P[1] - rho[0] * g * (-alt[0] - alt[1]))
        pt = (P[-2] + (P[-1] - P[-2]) / (alt[-1] - alt[-2]) * (2 * alth[-1] - alt[-1] - alt[-2]))
        ph = torch.cat([ps[None], self.up(P), 0.5 * (P[-1] + pt.clamp(min=0.0))[None]])
        th = torch.cat([T[:1], self.up(T), T[-1:]])
        ts = r["n_sw"] * r["kappa_sw"] * (P / p["P_Ref"]) ** (r["n_sw"] - 1) * rho * self.dz
        tl = (r["kappa_lw"] * (1 + r["n_lw"] * (1 - r["f_lw"]) / r["f_lw"]
                               * (P / p["P_Ref"]) ** (r["n_lw"] - 1)) * rho * self.dz)
        mu = torch.where(cz > 0, cz, torch.ones_like(cz))
        sw = [insol * (1 - r["albedo"]) * torch.exp(-r["kappa_sw"] / g * ph[-1] / mu)]
        for l in range(nv - 1, -1, -1):
            sw.append(sw[-1] * torch.exp(-ts[l] / mu))
        sw = torch.stack(sw[::-1])
        bc, da = 5.677036E-8, r["diff_ang"]
        bh, bl = bc * th ** 4, bc * T ** 4
        h = tl / 2
        ex = torch.exp(-h / da)

        def src(b0, bm, b1):
            e1 = b0 - bm + (bm - da / h * (b0 - bm)) * (1 - ex)
            e2 = bm - b1 + (b1 - da / h * (bm - b1)) * (1 - ex)
            s1, s2, sgn, fac = 0, 0, 1.0, 1.0
            for i in range(5):
                fac *= i + 2
                s1 = s1 + sgn * ((bm + (i + 1) * bm) / fac) * (h / da) ** (i + 1)
                s2 = s2 + sgn * ((b1 + (i + 1) * b0) / fac) * (h / da) ** (i + 1)
                sgn = -sgn
            thick = tl >= 1e-10
            return torch.where(thick, e1, s1) + torch.where(thick, e2, s2) * ex

        ed, eu, tr = src(bh[:-1], bl, bh[1:]), src(bh[1:], bl, bh[:-1]), torch.exp(-tl / da)
        dn = [torch.zeros_like(cz)]
        for l in range(nv - 1, -1, -1):
            dn.append(ed[l] + dn[-1] * tr[l])
        dn = torch.stack(dn[::-1])
        upw = [bc * r["Tint"] ** 4 + dn[0]]
        for l in range(nv):
            upw.append(eu[l] + upw[-1] * tr[l])
        upw = torch.stack(upw)
        net = upw - dn - sw
        heat = -(net[1:] - net[:-1]) / self.dz
        self.raw_heat = heat
        over = self.pr + self.Rd / (self.Cp - self.Rd) * heat * dt < 0
        heat = torch.where(over, -self.pr / dt, heat)
        self.Qheat = self.Qheat + heat
        top = ((p["A"] + alth[-1]) / p["A"]) ** 2 if self.case["deep"] else 1.0
        self.rt_out = dict(flw_up=upw, flw_dn=dn, fsw_dn=sw, tau=torch.cat([ts, tl]),
                           insol=insol[None], ASR=(sw[-1] * self.areasT * top)[None],
                           OLR=(upw[-1] * self.areasT * top)[None], cos_zenith=cz)

    # -- Thor --
    def thor(self):
        p, nv, N = self.p, self.nv, self.N
        Rd, Cp, g, A, dtl = self.Rd, self.Cp, p["Gravit"], p["A"], p["timestep"]
        Cv = Cp - Rd
        deep, nonh, eeq = self.case["deep"], self.case["nonhydro"], self.case["energy"]
        alt, alth, fr = self.alt, self.alth, self.fr
        M, W, Wc, rho, pr = self.Mh, self.Wh, self.W, self.Rho, self.pr
        Ms, rs_, ps_, Ws = (torch.zeros_like(q) for q in (M, rho, pr, W))
        pref = p["P_Ref"]
        dzc = alt[1:] - alt[:-1]
        pole = self.pole
        extr = (2 * alth[-1] - alt[-1] - alt[-2]) / (alt[-1] - alt[-2])
        extb = (alth[0] - alt[1]) / (alt[1] - alt[0])
        for rk in range(3):
            dt = dtl / 3 if rk == 0 else dtl / 6
            # advection and Coriolis
            v = M / rho + (Wc / rho) * fr[:, None]
            flux = [0, 0, 0]
            for j in range(7):
                mv, vv = (M, v) if j == 0 else (self.at(M, self.nb[j - 1]), self.at(v, self.nb[j - 1]))
                for c in range(3):
                    for k in range(3):
                        flux[c] = flux[c] + self.rs * self.div[j, k] * vv[c] * mv[k]
            adv = torch.stack(flux)
            del flux, mv, vv
            vw = torch.stack([self.pad(self.up(v[c]) * W[1:-1]) for c in range(3)])
            adv = adv + (vw[:, :-1] * self.r2h[:-1] - vw[:, 1:] * self.r2h[1:]) / (-self.dz * self.r2c)
            om = 2 * p["Omega"]
            if deep:
                adv = adv + torch.stack([-om * v[1] * rho, om * v[0] * rho, 0 * rho])
            else:
                adv = adv + torch.stack([om * (v[2] * fr[2] * fr[1] - v[1] * fr[2] ** 2) * rho,
                                         -om * (v[2] * fr[2] * fr[0] - v[0] * fr[2] ** 2) * rho,
                                         om * (v[1] * fr[2] * fr[0] - v[0] * fr[2] * fr[1]) * rho])
            # thermodynamics
            T = pr / (rho * Rd)
            h = Cv * T + pr / rho
            hh = torch.cat([h[:1], self.up(h), h[-1:]])
            pt = pref / (Rd * rho) * (pr / pref) ** (Cv / Cp)
            pth = torch.cat([(pt[1] + (pt[1] - pt[0]) * extb)[None], self.up(pt),
                             (pt[-2] + (pt[-1] - pt[-2]) * extr)[None]])
            rhoh, dpdz = self.up(rho), (pr[1:] - pr[:-1]) / dzc
            gb = -1 / (0.5 * (rho[0] + rho[1] + (rho[1] - rho[0]) * (-alt[0] - alt[1]) / dzc[0])) * (
                (pr[0] - (pr[1] - rho[0] * g * (-alt[0] - alt[1]))) / (2 * alt[0]))
            gt = -1 / (0.5 * (rho[-1] + rho[-2] + (rho[-1] - rho[-2]) * extr)) * (
                (pr[-2] - rho[-1] * g * (2 * alth[-1] - alt[-1] - alt[-2]) - pr[-1])
                / (2 * (alth[-1] - alt[-1])))
            gh = torch.cat([gb[None], -dpdz / rhoh, gt[None]])
            gw = self.pad(-(W[1:-1] / rhoh) * dpdz)
            cb = torch.cat([self.cb[1:], self.cb[-1:]])
            ca = torch.cat([self.ca[1:], self.ca[-1:]])
            gtil = gw[:-1] * cb + gw[1:] * ca
            if eeq:
                ep = g * alt + 0 * rho
                ek = 0.5 * ((M ** 2).sum(0) + Wc ** 2) / rho ** 2
                et = rho * (ep + ek) + Cv / Rd * pr
                eph = torch.cat([(g * alth[0] + 0 * rho[0])[None], self.up(ep),
                                 (g * alth[-1] + 0 * rho[0])[None]])
                ekh = torch.cat([(ek[1] + (ek[1] - ek[0]) * extb)[None], self.up(ek),
                                 (ek[-2] + (ek[-1] - ek[-2]) * extr)[None]])
                cen, face = h + ep + ek, hh + eph + ekh
            else:
                cen, face = pt, pth
            # hyperdiffusion
            args = [rho, M[0] / rho, M[1] / rho, M[2] / rho, Wc / rho, (Cv if eeq else Rd) * T]
            n = p["HyDiffOrder"] // 2
            for i in range(n):
                if i == n - 1 and i > 0:
                    args = [args[0]] + [a * rho for a in args[1:]]
                args = [self.laplacian(a) for a in args]
            args = [-self.kdh * (-1.0) ** n * a for a in args]
            drho, dM, dW, dp = args[0], self.tangent(torch.stack(args[1:4])), args[4], args[5]
            # slow modes
            damp = lambda mm, ww: -self.kdz * self.tangent(self.graddiv(self.graddiv(mm, ww)))  # noqa: E731
            damped = damp(M, W)
            advr = (adv * fr[:, None]).sum(0)
            adv = adv - advr * fr[:, None]
            if not nonh:
                advr = (M ** 2).sum(0) / (rho * (alt + A))
            gp = self.gradient(pr)
            gpt = self.tangent(gp)
            sM = -gpt - adv + damped + dM
            r2t, r2b, r2c = self.r2h[1:], self.r2h[:-1], self.r2c
            thick = torch.where(pole, self.dz * r2c, self.dr2dz)
            Wb = torch.cat([torch.zeros_like(W[:1]), W[1:]])
            srho = -(self.rs * self.stencil(self.div, M) + (Wb[1:] * r2t - Wb[:-1] * r2b) / thick) + drho
            hflux = self.rs * self.stencil(self.div, M * h)
            dwh = (Wb[1:] * r2t * hh[1:] - Wb[:-1] * r2b * hh[:-1]) / (self.dz * r2c)
            vgp = (gpt * M).sum(0) / rho
            sp = Rd / Cv * (-hflux - gtil - dwh + vgp + self.Qheat) + (Rd / Cv * dp if eeq else dp)
            grav = rho * g + (advr if deep else 0)
            sW = self.up(grav) + dpdz
            if nonh:
                sW = sW - self.up(dW)
            sW = self.pad(-sW)
            if rk > 0:
                Ms = self.tangent(self.Mh - M)
                rs_, ps_ = self.Rho - rho, self.pr - pr
                Ws = self.pad((self.Wh - W)[1:-1])
            # small steps
            for _ in range((1, 3, 6)[rk]):
                Ms = Ms + self.tangent((-self.gradient(ps_) + sM + damp(Ms, Ws)) * dt)
                Fr = self.rs * self.stencil(self.div, Ms)
                Fp = self.rs * self.stencil(self.div, (Ms + M) * cen)
                Sp = -(Rd / Cv) * (self.rs * self.stencil(self.div, Ms * h)) + sp
                Sd = -Fr + srho
                cr, gc = Cv / (Rd * dt * dt), g * Cv / Rd
                lo, hi = (alt[1:] - alth[1:-1]) / dzc, (alth[1:-1] - alt[:-1]) / dzc
                CR, GC = cr[:-1] * lo + cr[1:] * hi, gc[:-1] * lo + gc[1:] * hi
                dzp, dzh, dzm = 1 / (alth[2:] - alth[1:-1]), 1 / dzc, 1 / (alth[1:-1] - alth[:-2])
                il, im = (alt[1:] - alth[1:-1]) * dzp * dzh, -(alt[:-1] - alth[1:-1]) * dzm * dzh
                if deep:
                    o2, t3 = (alth[1:-1] + A) ** -2, 2 * (alth[1:-1] + A) ** -3
                    H = hh * self.r2h
                else:
                    o2, t3, H = 1.0, 0.0, hh
                c_ = -dzp * dzh * o2 * H[2:] - im * (gh[2:] + GC - t3 * H[2:])
                b_ = (CR if nonh else 0) + dzh * (dzp + dzm) * o2 * H[1:-1] + (il - im) * (
                    gh[1:-1] + GC - t3 * H[1:-1])
                a_ = -dzm * dzh * o2 * H[:-2] + il * (gh[:-2] + GC - t3 * H[:-2])
                d_ = -CR * ((-Ws[1:-1] if nonh else 0) + dt * dt * (Sp[1:] - Sp[:-1]) * dzh
                            + dt * dt * g * self.up(Sd) + g * dt * self.up(rs_)
                            + dt * (ps_[1:] - ps_[:-1]) * dzh - dt * sW[1:-1])
                cc, dd = [c_[0] / b_[0]], [d_[0] / b_[0]]
                for l in range(1, nv - 1):
                    t = 1 / (b_[l] - cc[-1] * a_[l])
                    dd.append((d_[l] - dd[-1] * a_[l]) * t)
                    cc.append(c_[l] * t)
                w = [dd[-1]]
                for l in range(nv - 3, -1, -1):
                    w.append(dd[l] - cc[l] * w[-1])
                Ws = self.pad(torch.stack(w[::-1]))
                Wt = Ws + W
                Wt = torch.cat([torch.zeros_like(W[:1]), Wt[1:]])
                dwdz = (Ws[1:] * r2t - Ws[:-1] * r2b) / thick
                dwp = (Wt[1:] * face[1:] * r2t - Wt[:-1] * face[:-1] * r2b) / (self.dz * r2c)
                aux = -(Fp + dwp) * dt
                rold = rho + rs_
                rs_new = rs_ + (srho - Fr - dwdz) * dt
                if eeq:
                    et = et + aux + dp * dt + self.Qheat * dt
                    wc = (Wt[:-1] * (alth[1:] - alt) + Wt[1:] * (alt - alth[:-1])) / self.dz
                    rn = rho + rs_new
                    kin = 0.5 * (((Ms + M) ** 2).sum(0) + wc ** 2) / rn
                    ps_ = Rd / Cv * (et - rn * g * alt - kin) - pr
                else:
                    th = pref / (Rd * rold) * ((ps_ + pr) / pref) ** (Cv / Cp)
                    pn = pref * (Rd * (aux + th * rold) / pref) ** (Cp / Cv)
                    ps_ = pn - pr + dp * dt + Rd / Cv * self.Qheat * dt
                rs_ = rs_new
            M, rho, pr = self.tangent(M + Ms), rho + rs_, pr + ps_
            W = self.pad((W + Ws)[1:-1])
            Wc = W[:-1] * self.cb + W[1:] * self.ca
        # the temperature a step leaves is the last stage's (computed from its start)
        self.Mh, self.Wh, self.W, self.Rho, self.pr, self.T = M, W, Wc, rho, pr, T

    def fields(self, names):
        d = dict(Rho=self.Rho, pressure=self.pr, Mh=self.Mh.reshape(-1, self.N), Wh=self.Wh, W=self.W,
                 temperature=self.T, profx_Qheat=self.Qheat)
        if self.case["rt"] and hasattr(self, "rt_out"):
            d.update(self.rt_out)
        return {n: d[n] for n in names}

    def host(self, names):
        """The reference layouts a host program holds."""
        d = dict(Rho=self.Rho.t(), pressure=self.pr.t(), Mh=self.Mh.permute(2, 1, 0), Wh=self.Wh.t())
        return {n: d[n].contiguous().cpu().numpy().reshape(-1) for n in names}

    def globdiag(self):
        p, A, deep = self.p, self.p["A"], self.case["deep"]
        zu, zl = self.alth[1:] + A, self.alth[:-1] + A
        vol = self.areasT / A ** 2 * (zu ** 3 - zl ** 3) / 3 if deep else self.areasT * (zu - zl)
        lon, lat = self.lon, self.lat
        r = torch.stack([torch.cos(lat) * torch.cos(lon), torch.cos(lat) * torch.sin(lon),
                         torch.sin(lat)])
        ek = 0.5 * ((self.Mh + self.W * r[:, None]) ** 2).sum(0) / self.Rho
        E = (ek + (self.Cp - self.Rd) * self.T * self.Rho + self.Rho * p["Gravit"] * self.alt) * vol
        R = A + self.alt
        x = [R * self.fr[k] for k in range(3)]
        M, q = self.Mh, self.Rho * p["Omega"] * R
        am = [x[1] * M[2] - x[2] * M[1] - q * x[2] * torch.cos(lat) * torch.cos(lon),
              -x[0] * M[2] + x[2] * M[0] - q * x[2] * torch.cos(lat) * torch.sin(lon),
              x[0] * M[1] - x[1] * M[0] + q * R * torch.cos(lat) ** 2]
        s = self.Cp * torch.log(self.T * (p["P_Ref"] / self.pr) ** (self.Rd / self.Cp))
        total = lambda a: math.fsum((a * vol).reshape(-1).cpu().tolist())  # noqa: E731
        return dict(energy=math.fsum(E.reshape(-1).cpu().tolist()), mass=total(self.Rho),
                    am=np.array([total(a) for a in am]), entropy=total(s))


def _mix(z):
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _train_exact(case, seed, e):
    """The Adam steps in 64 bits on the batches the seed selects (features and targets as logged)."""
    e.profx()
    X = torch.cat([e.T.t(), torch.log(e.pr_before.t()), e.rt_out["cos_zenith"][:, None]], 1)
    Y = (e.raw_heat / (e.Rho * (e.Cp - e.Rd))).t()
    X, Y = X.float().double(), Y.float().double()
    norm = lambda a: (a.mean(0), torch.where((s := a.std(0, unbiased=False)) > 0, s, 1 + 0 * s))  # noqa: E731
    (xm, xs), (ym, ys) = norm(X), norm(Y)
    X, Y = (X - xm) / xs, (Y - ym) / ys
    N, nv = X.shape[0], case["nv"]
    layers = [[torch.as_tensor(W, device=DEV).double(), torch.as_tensor(b, device=DEV).double()]
              for W, b in _layers(case, seed)]
    X = torch.nn.functional.pad(X, (0, layers[0][0].shape[1] - X.shape[1]))
    par = [q.requires_grad_() for l in layers for q in l]
    mom = [[torch.zeros_like(q), torch.zeros_like(q)] for q in par]
    losses = []
    for t in range(1, ADAM_STEPS + 1):
        with np.errstate(over="ignore"):
            s = np.uint64(1 + seed) ^ (np.uint64(0xD1B54A32D192ED03) * np.uint64(t))
            z = _mix(s + np.uint64(0x9E3779B97F4A7C15) * np.arange(1, BATCH + 1, dtype=np.uint64))
        u = (z >> np.uint64(11)).astype(np.float64) * 2.0 ** -53
        rows = torch.as_tensor((u * N).astype(np.int64) % N, device=DEV)
        a = X[rows]
        for l in range(3):
            a = torch.nn.functional.gelu(a @ par[2 * l].t() + par[2 * l + 1], approximate="tanh")
        out = (a @ par[6].t() + par[7])[:, :nv]
        loss = ((out - Y[rows]) ** 2).mean()
        losses.append(float(loss.detach()))
        grads = torch.autograd.grad(loss, par)
        with torch.no_grad():
            for q, m, gq in zip(par, mom, grads):
                m[0].mul_(0.9).add_(0.1 * gq)
                m[1].mul_(0.999).add_(0.001 * gq * gq)
                q -= ADAM_LR * (m[0] / (1 - 0.9 ** t)) / ((m[1] / (1 - 0.999 ** t)).sqrt() + 1e-8)
    par = [q.detach().cpu().numpy() for q in par]
    return [[par[2 * l], par[2 * l + 1]] for l in range(4)] + [np.array([losses[0], losses[-1]])]


def exact(case, seed):
    e = _Exact(case, _inputs(case, seed))
    e.pr_before = e.pr
    call = case["call"]
    if call == "step":
        e.profx()
        e.thor()
        return e.fields(STATE_OUT)
    if call == "thor":
        e.thor()
        return e.fields(STATE_OUT)
    if call == "profx":
        e.profx()
        return e.fields(["pressure", "Mh", "W", "temperature", "profx_Qheat"]
                        + (RT_OUT if case["rt"] else []))
    if call == "exchange":
        e.profx()
        e.thor()
        return e.host(STATE_IO)
    if call == "globdiag":
        return e.globdiag()
    return _train_exact(case, seed, e)
