"""The plane kernels (256-column tiles staged level by level) and the column kernels of the step, where
they can go wrong: level counts at the edges of the level chunks and of the CTAs' ranges, each model form,
deviations beyond the pressure series, grids whose tiles are not rhombi of 16 x 16 (which the
column-tile kernels serve), and stage arrays that a caller looks at.

Against the CPU restatement, and for other rhombi against the plane kernels on the same columns. The
tolerance of a field is 1e-12 of its maximum (density, pressure, temperature), and for the momenta the
rounding of the terms they are small residuals of: the hydrostatic terms rho g dt enter each of the ten
small steps with one rounding each of a few operations, so 64 units of 2^-53 rho g dt cover both sides.
"""
import ctypes

import numpy as np
import pytest

import thor_b200
from thorx_testlib import (RT_WASP43B, Oracle, STATE_FIELDS, grid_dict, hot_jupiter_params, initial_state,
                           make_params, rel_err, thorx_params)

TIGHT = {"Rho", "pressure", "temperature"}
FIELDS = STATE_FIELDS + ["temperature"]


def windy(g, c, nv, amp):
    """The seeded rest state with a zonal wind of 10 m/s."""
    ic = initial_state(g, g.point_num, nv, c, amp=amp)
    lon, lat = g["lonlat"][0::2], g["lonlat"][1::2]
    rho = ic["Rho"].reshape(-1, nv)
    east = np.stack([-np.sin(lon), np.cos(lon), 0 * lon], 1) * np.cos(lat)[:, None]
    ic["Mh"] = (10.0 * rho[:, :, None] * east[:, None, :]).reshape(-1)
    return ic


def tolerance(field, ref, ic, c, dt):
    if field in TIGHT:
        return 1e-12
    return max(1e-12, 64 * 2.0 ** -53 * ic["Rho"].max() * c["Gravit"] * dt / np.abs(ref).max())


def run_product(g, glevel, c, dt, ic, nsteps=1, precision=0, escape=(), grid=None):
    x = thor_b200.Thorx(grid if grid is not None else grid_dict(g), glevel,
                        thorx_params(c, dt, precision=precision))
    for k, v in ic.items():
        x.set(k, v)
    for f in escape:
        x.device_field(f)
    x.step(nsteps)
    x.sync()
    out = {f: x.get(f) for f in FIELDS}
    out["thomas"] = x.check_thomas(1e-8)[0]
    x.close()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("nv,over,amp", [
    (3, {}, 0.1), (7, {}, 0.1), (8, {}, 0.1), (9, {}, 0.1), (33, {}, 0.1), (128, {}, 0.1),
    (17, dict(DeepModel=0, NonHydro=0), 0.1),
    (16, dict(energy_equation=1, GravHeightVar=1), 0.1),
    (12, dict(DivDampP=0, HyDiffOrder=2), 0.1),
    (12, dict(HyDiffOrder=6), 0.1),
    (12, dict(HyDiff=0, held_suarez=0), 0.1),
    (12, {}, 60.0),  # +-60 K: pressure deviations above the series' 1/32, the general form
])
def test_step_matches_the_cpu_restatement(nv, over, amp):
    glevel, dt = 4, 300.0
    p, c = make_params(glevel, dt, **over)
    g = thor_b200.Icogrid(glevel, nv)
    ic = windy(g, c, nv, amp)
    got = run_product(g, glevel, c, dt, ic)
    o = Oracle(g, p)
    for k, v in ic.items():
        o.set(k, v)
    o.step(1)
    bad = {}
    for f in FIELDS:
        ref = o.get(f)
        err, tol = rel_err(got[f], ref), tolerance(f, ref, ic, c, dt)
        # the larger state's own terms are larger by the relative size of its deviations
        if not (np.isfinite(got[f]).all() and err <= tol * (10.0 if amp > 1.0 else 1.0)):
            bad[f] = (err, tol)
    o.close()
    assert not bad, bad
    # the solve's rows are kept for the check (its own test holds the residuals to the reference's bound,
    # relative to right-hand sides that may pass through zero here)
    assert got["thomas"] > 0.0


RT_FLUXES = ["cos_zenith", "insol", "insol_ann", "ASR", "OLR", "fsw_dn", "flw_up", "flw_dn", "tau", "phtemp",
             "thtemp"]


@pytest.mark.gpu
@pytest.mark.parametrize("nv,rt", [
    (20, {}), (7, {}), (128, {}),
    (9, dict(sync_rot=0, mean_motion=2.0e-5, ecc=0.3, obliquity=23.0, longp=40.0, alpha_i=5.0)),
    (33, dict(n_sw=2.0, n_lw=1.5, latf_lw=1, kappa_lw_pole=0.004)),
    (8, dict(rt1Dmode=1, n_sw=1.7)),
    (7, dict(kappa_lw=1e-17, kappa_lw_pole=1e-17)),  # every layer optically thin: the source's series
])
def test_radiative_transfer_matches_the_cpu_restatement(nv, rt):
    glevel, dt = 4, 300.0
    rt = dict(RT_WASP43B, **rt)
    p, c = hot_jupiter_params(glevel, dt)
    g = thor_b200.Icogrid(glevel, nv, A=c["A"], Top_altitude=c["Top_altitude"])
    x, o = thor_b200.Thorx(grid_dict(g), glevel, thorx_params(c, dt)), Oracle(g, p)
    for k, v in initial_state(g.arrays, g.point_num, nv, c, amp=1.0).items():
        x.set(k, v), o.set(k, v)
    x.rt_enable(rt), o.rt(rt)
    for _ in range(2):  # the second with an orbit that has moved on
        x.profx()
        x.sync()
        o.step(1, profx=True, thor=False)
    got = {f: (x.get(f), o.get(f)) for f in RT_FLUXES + ["dtemp", "profx_Qheat", "pressure", "temperature"]}
    x.close(), o.close()
    # a flux is a sum of up to nv positive terms, each of a few transcendental functions of two units
    # each; a cell's heating is the difference of the fluxes at its two interfaces over its height
    flux = max(np.abs(got[f][1]).max() for f in ("fsw_dn", "flw_up", "flw_dn"))
    dz = np.diff(np.asarray(g["Altitudeh"])).min()
    for f, (a, b) in got.items():
        tol = 4e-12 * flux / dz if f in ("dtemp", "profx_Qheat") else 1e-12 * np.abs(b).max()
        assert np.isfinite(b).all() and np.abs(a - b).max() <= tol, (f, np.abs(a - b).max(), tol)


def smaller_rhombi(g, nl=8, shuffle=None):
    """The same grid with every rhombus of 16 x 16 cut into rhombi of nl x nl, its columns (all but the
    poles) in a random order with shuffle, a seed: (grid, old column of each new one)."""
    d = grid_dict(g)
    N, old, nr, k = g.point_num, g.nl_region, g.nr, g.nl_region // nl
    m = np.asarray(g["maps"]).reshape(nr, old + 2, old + 2)
    maps, order = [], []
    for r in range(nr):
        for by in range(k):
            for bx in range(k):
                w = m[r, by * nl:by * nl + nl + 2, bx * nl:bx * nl + nl + 2]
                maps.append(w)
                order.append(w[1:-1, 1:-1].reshape(-1))
    order = np.concatenate(order)
    if shuffle is not None:
        np.random.default_rng(shuffle).shuffle(order)
    order = np.concatenate([order, [N - 2, N - 1]])
    new = np.empty(N, np.int32)
    new[order] = np.arange(N, dtype=np.int32)
    relabel = lambda a: np.where(a >= 0, new[np.maximum(a, 0)], a).astype(np.int32)  # noqa: E731
    out = dict(d, nl_region=nl, nr=nr * k * k, maps=relabel(np.stack(maps)).reshape(-1))
    for name in ("lonlat", "areas", "areasTr", "areasT", "nvecoa", "nvecti", "nvecte", "div", "grad",
                 "func_r"):
        a = np.asarray(d[name])[:N * (len(d[name]) // N)].reshape(N, -1)
        out[name] = np.ascontiguousarray(a[order]).reshape(-1)
    out["point_local"] = relabel(np.asarray(d["point_local"]).reshape(N, 6)[order]).reshape(-1)
    return out, order


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [thor_b200.FP64, thor_b200.MIXED])
def test_other_rhombi_give_the_same_step(precision):
    """Columns grouped in rhombi of 8 x 8 take the column-tile kernels: the same step on the same columns."""
    glevel, nv, dt = 4, 13, 300.0
    p, c = make_params(glevel, dt)
    g = thor_b200.Icogrid(glevel, nv)
    ic = windy(g, c, nv, 0.1)
    ref = run_product(g, glevel, c, dt, ic, precision=precision)
    grid, order = smaller_rhombi(g)
    N = g.point_num
    got = run_product(g, glevel, c, dt,
                      {k: v.reshape(N, -1)[order].reshape(-1) for k, v in ic.items()},
                      precision=precision, grid=grid)
    for f in FIELDS:
        a = np.empty_like(got[f]).reshape(N, -1)
        a[order] = got[f].reshape(N, -1)
        err, tol = rel_err(a.reshape(-1), ref[f]), tolerance(f, ref[f], ic, c, dt)
        # mixed: the column-tile form's FP32 stencils, 2^-24 of the damping and diffusion tendencies
        assert err <= (tol if precision == thor_b200.FP64 else 1e-7), (f, err, tol)


@pytest.mark.gpu
def test_stage_arrays_handed_out_are_kept_and_change_nothing():
    glevel, nv, dt = 4, 10, 600.0
    p, c = make_params(glevel, dt)
    g = thor_b200.Icogrid(glevel, nv)
    ic = windy(g, c, nv, 0.1)
    ref = run_product(g, glevel, c, dt, ic, nsteps=3)
    got = run_product(g, glevel, c, dt, ic, nsteps=3, escape=("Mhk", "Rhok", "profx_dMh"))
    for f in FIELDS:
        assert np.array_equal(got[f], ref[f]), f


@pytest.mark.gpu
@pytest.mark.parametrize("nl", [8, 16])
def test_columns_in_any_order_give_the_same_step(nl):
    """Columns in a random order: a tile of 256 has more neighbours outside it (about 1000 here) than the
    ring of a grid with neighbourhood holds, and a rhombus of 16 x 16 is no tile."""
    glevel, nv, dt = 4, 9, 300.0
    p, c = make_params(glevel, dt)
    g = thor_b200.Icogrid(glevel, nv)
    ic = windy(g, c, nv, 0.1)
    N, out = g.point_num, []
    for cut in (dict(nl=8), dict(nl=nl, shuffle=5)):
        grid, order = smaller_rhombi(g, **cut)
        got = run_product(g, glevel, c, dt,
                          {k: v.reshape(N, -1)[order].reshape(-1) for k, v in ic.items()}, grid=grid)
        out.append({f: np.empty_like(got[f]).reshape(N, -1) for f in FIELDS})
        for f in FIELDS:
            out[-1][f][order] = got[f].reshape(N, -1)
    if nl == 16:  # as many outside neighbours as said
        pl = grid["point_local"].reshape(N, 6)[:256]
        assert len(set(pl[pl >= 256].tolist())) > 768
    for f in FIELDS:
        assert np.array_equal(out[0][f], out[1][f]), f


@pytest.mark.gpu
def test_a_missing_neighbour_reads_zero():
    """A rhombus whose map lacks a halo entry (-1: a hole, whose fields read 0): no triangles with that
    neighbour exist, so the column-tile kernels serve the grid, in rhombi of 16 x 16 as in smaller ones."""
    glevel, nv, dt = 4, 9, 300.0
    p, c = make_params(glevel, dt)
    g = thor_b200.Icogrid(glevel, nv)
    maps = np.array(g["maps"]).reshape(g.nr, 18, 18)
    maps[3, 9, 17] = -1  # beyond the edge of columns (15, 7) and (15, 8)
    g.arrays["maps"] = maps.reshape(-1)
    ic = windy(g, c, nv, 0.1)
    ref = run_product(g, glevel, c, dt, ic)
    grid, order = smaller_rhombi(g)
    N = g.point_num
    got = run_product(g, glevel, c, dt,
                      {k: v.reshape(N, -1)[order].reshape(-1) for k, v in ic.items()}, grid=grid)
    for f in FIELDS:
        a = np.empty_like(got[f]).reshape(N, -1)
        a[order] = got[f].reshape(N, -1)
        # the same kernels on the same columns in another order
        assert np.isfinite(ref[f]).all() and np.array_equal(a.reshape(-1), ref[f]), f


@pytest.mark.gpu
def test_no_memory_for_the_other_form():
    """A grid holds the weights of the kernels that serve it: the plane kernels' 42 doubles a column and the
    triangles of the tiles' edges, or the column-tile kernels' 84 doubles and floats."""
    import torch
    glevel, nv = 5, 4
    p, c = make_params(glevel, 300.0)
    g = thor_b200.Icogrid(glevel, nv, spring=False)
    held = []
    for grid in (grid_dict(g), smaller_rhombi(g)[0]):
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        x = thor_b200.Thorx(grid, glevel, thorx_params(c, 300.0))
        held.append(free - torch.cuda.mem_get_info()[0])
        x.close()
    assert held[0] < held[1], held


def count_kernels(x, stream):
    """Kernel nodes of one step, captured from the calls of thorx_step without its own graph."""
    import torch
    from cuda.bindings import runtime as rt
    thor_b200.lib().thorx_set_graph_mode(x.h, 0)
    x.step(1)
    x.sync()

    def ok(r):
        assert r[0] == rt.cudaError_t.cudaSuccess, r[0]
        return r[1:] if len(r) > 2 else r[-1]

    ok(rt.cudaStreamBeginCapture(stream.cuda_stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal))
    x.step(1)
    graph = ok(rt.cudaStreamEndCapture(stream.cuda_stream))
    n = ok(rt.cudaGraphGetNodes(graph, 0))[1]
    nodes = ok(rt.cudaGraphGetNodes(graph, n))[0]
    kinds = [ok(rt.cudaGraphNodeGetType(k)) for k in nodes]
    ok(rt.cudaGraphDestroy(graph))
    torch.cuda.synchronize()
    return kinds.count(rt.cudaGraphNodeType.cudaGraphNodeTypeKernel)


class ModuleC(ctypes.Structure):
    _fields_ = [("user", ctypes.c_void_p)] + [(h, ctypes.c_void_p) for h in (
        "init", "slow", "fast", "end", "phy")]


FAST_HOOK = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p,
                             ctypes.c_int, ctypes.c_int, ctypes.c_double)(lambda *a: 0)


@pytest.mark.gpu
@pytest.mark.parametrize("over,what", [
    ({}, ""), ({}, "8x8"), ({}, "module"), ({}, "fast"), ({}, "8x8 module"), ({}, "8x8 fast"),
    (dict(HyDiffOrder=6, energy_equation=1), ""), (dict(HyDiff=0), ""), (dict(DivDampP=0), "module"),
    (dict(HyDiffOrder=2), "mixed"), ({}, "sponge0"), ({}, "sponge1"), ({}, "sponge2 vertical"), ({}, "rt"),
    ({}, "rt log"), ({}, "rt use"), ({}, "rt use_log")])
def test_kernels_per_step_is_what_a_step_launches(over, what):
    import torch
    glevel, nv, dt = 4, 8, 300.0
    p, c = make_params(glevel, dt, **over)
    g = thor_b200.Icogrid(glevel, nv, spring=False)
    stream = torch.cuda.Stream()
    x = thor_b200.Thorx(smaller_rhombi(g)[0] if "8x8" in what else grid_dict(g), glevel,
                        thorx_params(c, dt, precision=int("mixed" in what)), stream=stream.cuda_stream)
    x.init_rest_state(300.0)
    if "module" in what or "fast" in what:
        m = ModuleC(fast=ctypes.cast(FAST_HOOK, ctypes.c_void_p) if "fast" in what else None)
        assert thor_b200.lib().thorx_module_add(ctypes.c_void_p(x.h), ctypes.byref(m)) == 0
    if "sponge" in what:
        x.sponge(dict(raysp_calc_mode=int(what[6])))
    if "vertical" in what:
        x.vert_hydiff(0.001, 6)
    if "rt" in what:
        x.rt_enable(RT_WASP43B)
    if "log" in what or "use" in what:
        x.sur_create(hidden=256, train_batch=128, log_capacity=4096)
        n_in = 2 * nv + 1
        x.sur_set_normalisation(*[np.full(n, v, np.float32) for n, v in ((n_in, 0), (n_in, 1), (nv, 0), (nv, 1))])
        x.sur_mode(dict(log=1, use=2, use_log=3)[what.split()[1]])
    assert x.kernels_per_step() == count_kernels(x, stream)
    # each class of a kernel the step launches has bytes and launches
    for name, nbytes, launches in x.kernel_table():
        assert (launches > 0) == (nbytes > 0) or launches == 0, (name, nbytes, launches)
    x.close()


STAGE = {"Mhk": "Mh", "Rhok": "Rho", "pressurek": "pressure", "Whk": "Wh", "Wk": "W"}


def packed(x, field, N, levels, comps):
    """A field's columns by thorx_pack_columns, in the order of Thorx.get."""
    import torch
    cols = torch.arange(N, dtype=torch.int32, device="cuda")
    buf = torch.zeros(N, comps, levels, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    x._check(thor_b200.lib().thorx_pack_columns(x.h, field.encode(), cols.data_ptr(), N, buf.data_ptr()))
    x.sync()
    return buf.permute(0, 2, 1).cpu().numpy().reshape(-1)


@pytest.mark.gpu
@pytest.mark.parametrize("first", ["before", "after"])  # the handing out of a device pointer
def test_stage_arrays_hold_the_end_of_the_dynamics(first):
    """Between calls the stage arrays are the state at the end of the last thorx_thor (which a following
    thorx_profx leaves alone), bit for bit, however they are read."""
    import torch
    glevel, nv, dt = 4, 10, 600.0
    p, c = make_params(glevel, dt)
    g = thor_b200.Icogrid(glevel, nv)
    N = g.point_num
    x, y = (thor_b200.Thorx(grid_dict(g), glevel, thorx_params(c, dt)) for _ in range(2))
    for k, v in windy(g, c, nv, 0.1).items():
        x.set(k, v)
    cols = torch.arange(N, dtype=torch.int32, device="cuda")
    shape = {k: (nv + (k == "Whk"), 3 if k == "Mhk" else 1) for k in STAGE}

    def check(want, ctx, how):
        for k in STAGE:
            got = packed(ctx, k, N, *shape[k])
            assert np.array_equal(got, want[k]), (how, k)

    def state():
        return {k: x.get(v) for k, v in STAGE.items()}

    if first == "before":
        for k in STAGE:
            x.device_field(k)
    x.step(2)
    x.sync()
    check(state(), x, "step")
    for k in STAGE:
        y.copy_columns(x, k, cols.data_ptr(), N)
    y.sync()
    check(state(), y, "copied")
    x.thor()
    want = state()
    x.profx()
    if first == "after":
        for k in STAGE:
            x.device_field(k)
    check(want, x, "thor, profx")
    assert not np.array_equal(x.get("Mh"), want["Mhk"])  # the forcing has moved the state on
    x.step(1)
    x.sync()
    check(state(), x, "step again")
    x.close(), y.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nv", [3, 8, 48])
def test_globdiag_chunks(nv):
    """The chunked global sums against sums of their own per-cell terms (math.fsum: exact)."""
    import math
    glevel, dt = 4, 600.0
    p, c = make_params(glevel, dt)
    g = thor_b200.Icogrid(glevel, nv)
    x = thor_b200.Thorx(grid_dict(g), glevel, thorx_params(c, dt))
    for k, v in windy(g, c, nv, 0.1).items():
        x.set(k, v)
    total, cells = x.globdiag_fields()
    assert list(total) == x.globdiag()
    for t, a in zip(total, cells):
        # compensated sums are rounded once; 2^-52 of the terms' magnitude covers a cancelling total
        assert abs(t - math.fsum(a.tolist())) <= 2.0 ** -52 * max(abs(t), 1e-12 * np.abs(a).sum())
    x.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nv", [8, 33, 57])
def test_globdiag_volumes_do_not_cancel(nv):
    """The volume of a cell is a difference of cubes of radii 2e2 to 1e4 times as large as the layer: every
    level's against rational arithmetic, to the few roundings of a form that does not cancel."""
    from fractions import Fraction as F
    glevel, dt = 4, 600.0
    p, c = make_params(glevel, dt)
    g = thor_b200.Icogrid(glevel, nv)
    x = thor_b200.Thorx(grid_dict(g), glevel, thorx_params(c, dt))
    for k, v in windy(g, c, nv, 0.1).items():
        x.set(k, v)
    N = g.point_num
    mass = x.globdiag_fields()[1][1].reshape(N, nv)
    rho, areasT = x.get("Rho").reshape(N, nv), np.asarray(g["areasT"])
    x.close()
    z = [F(float(a)) for a in np.asarray(g["Altitudeh"]) + c["A"]]
    for lev in range(nv):
        level = (z[lev + 1] ** 3 - z[lev] ** 3) / 3 / F(c["A"]) ** 2
        for col in (0, 777, N - 1):
            exact = F(float(rho[col, lev])) * F(float(areasT[col])) * level
            # twelve roundings of at most 2^-53: A^2, the area, dz, three products, two sums, three factors, / 3
            assert abs(F(float(mass[col, lev])) / exact - 1) <= 12 * F(1, 2 ** 53), (lev, col)
