// Double-gray radiative transfer (DualbandGray) and the insolation it needs, on the device.
//
// Reference: Insolation::phy_loop (src/ESP/insolation.cu:459-490, orbit update :514-529,
// calc_zenith :128-168) and radiative_transfer::phy_loop (spin-up/down, rtm_dual_band launch,
// annual insolation; src/physics/modules/src/radiative_transfer.cu:769-1105) with the kernel
// rtm_dual_band and its device functions (src/physics/modules/inc/profx_RT.h:30-587). The
// arithmetic of each piece follows the reference operation for operation.
//
// Differences of form: the orbit update, a few scalar lines of host code in the reference, runs
// in a one-thread kernel on a device-resident step counter so that a captured step graph
// advances it by itself; the column kernel works on the column-fastest layout (each level a
// plane, coalesced across a warp, the levels of a column spread over the warps of its CTA).
// GravHeightVar with RT is rejected at enable time: the reference's radcsw then reads
// Altitudeh[nv+1], past the end of the array (profx_RT.h:68).
#include "dyn_common.cuh"

namespace thorx {
namespace {

// Kepler's equation by the third-order iteration of insolation.cu:65-88 (which stops as soon as
// the last correction is not above 1e-15, signed); bounded at 100 iterations.
__device__ double solve_kepler(double M, double ecc) {
    double E  = M + (sin(M) < 0.0 ? -1.0 : 1.0) * 0.85 * ecc;
    double d3 = 1.0;
    for (int it = 0; it < 100 && d3 > 1e-15; it++) {
        double fi = E - ecc * sin(E) - M, f1 = 1.0 - ecc * cos(E), f2 = ecc * sin(E),
               f3 = ecc * cos(E);
        double d1 = -fi / f1;
        double d2 = -fi / (f1 + 0.5 * d1 * f2);
        d3        = -fi / (f1 + 0.5 * d2 * f2 + 1. / 6. * d2 * d2 * f3);
        E         = E + d3;
    }
    return E;
}

// Orbit update (when the reference calls it), spin-up/down scaling and the run flag of this step.
__global__ void rt_orbit_kernel(RtConst c, Phys P, RtStep* st) {
    step_begin();
    step_wait();
    const long long nstep = st->nstep;
    st->cur               = nstep;
    st->nstep             = nstep + 1;
    const double dt       = P.timestep;
    if (!c.sync_rot || c.ecc > 1e-10) {
        const double time = nstep * dt;
        double       M    = fmod((c.mean_motion * time + c.mean_anomaly_i), (2 * M_PI));
        double       E    = fmod(solve_kepler(M, c.ecc), (2 * M_PI));
        st->r_orb         = 1.0 - c.ecc * cos(E);
        double f          = 2.0 * atan(sqrt((1.0 + c.ecc) / (1.0 - c.ecc)) * tan(E / 2.0));
        if (f < 0.0)
            f += 2 * M_PI;
        const double true_long = fmod((f + c.longp), (2 * M_PI));
        st->sin_decl           = sin(c.obliquity) * sin(true_long);
        st->cos_decl           = sqrt(1.0 - st->sin_decl * st->sin_decl);
        st->alpha              = -P.Omega * time + true_long - c.true_long_i + c.alpha_i;
    }
    bool   run = true;
    double Qs  = 1.0;
    if (c.spinup_start > -1 && c.spinup_stop > -1) {
        if (nstep < c.spinup_start) {
            run = false;
            Qs  = 0.0;
        }
        else if (nstep >= c.spinup_start && nstep <= c.spinup_stop) {
            double x = (double)(nstep - c.spinup_start) / (double)(c.spinup_stop - c.spinup_start);
            Qs       = (1 + sin(M_PI * x - M_PI / 2.0)) / 2.0;
            run      = true;
        }
    }
    if (c.spindown_start > -1 && c.spindown_stop > -1) {
        if (nstep >= c.spindown_start && nstep <= c.spindown_stop) {
            double x = (double)(nstep - c.spindown_start) / (double)(c.spindown_stop - c.spindown_start);
            Qs       = 1.0 - (1 + sin(M_PI * x - M_PI / 2.0)) / 2.0;
            run      = true;
        }
        else if (nstep >= c.spindown_stop) {
            run = false;
            Qs  = 0.0;
        }
    }
    st->Qheat_scaling = Qs;
    st->run           = run;
}

// The source function of an optically thin layer (tau < 1e-10), source_func_lin's series
// (profx_RT.h:145-157): kept out of line, since hardly any layer takes it.
__device__ __noinline__ double source_thin(double bb, double bl, double bt, double h, double ex) {
    double e1 = 0.0, e2 = 0.0, sign = 1.0, fac = 1.0, hp = 1.0;
    for (int i = 0; i < 5; i++) {
        fac *= i + 2;
        hp *= h;
        e1 = e1 + sign * ((bl + (i + 1) * bl) / fac) * hp;
        e2 = e2 + sign * ((bt + (i + 1) * bb) / fac) * hp;
        sign = -sign;
    }
    return e1 + e2 * ex;
}
// source_func_lin (profx_RT.h:133-160) with q = diff_ang / (tau / 2) and ex = exp(-(tau / 2) / diff_ang),
// which the two directions of a layer share
__device__ __forceinline__ double source_func_lin(double bb, double bl, double bt, double q, double ex) {
    const double e1 = bb - bl + (bl - q * (bb - bl)) * (1.0 - ex);
    const double e2 = bl - bt + (bt - q * (bl - bt)) * (1.0 - ex);
    return e1 + e2 * ex;
}
// x^n; the opacity exponents n - 1 of the usual n = 1 and n = 2 need no pow
__device__ __forceinline__ double opacity_pow(double x, double n) {
    return n == 0.0 ? 1.0 : n == 1.0 ? x : pow(x, n);
}

// calc_zenith, the top-of-atmosphere insolation and annual_insol, then rtm_dual_band
// (profx_RT.h:316-587) with computetau, radcsw (no surface, GravHeightVar excluded), radclw
// (reflecting lower boundary), the cooling limiter and the coupling into profx_Qheat. The reference
// computes the insolation inside radcsw and the annual average after the RT; both depend on the
// zenith angle only, so computing them first changes no value.
//
// A CTA is 32 columns x 8 warps. What a level contributes (optical depths, transmissions, source
// terms: the exponentials) does not depend on the other levels and is computed level-parallel into
// shared memory; only the flux recurrences, one multiply-add per level, run down and up the column
// (the longwave ones on warp 0, the shortwave one on warp 1); then the heating and the stores are
// level-parallel again. A thread per column with every level in turn (80 CTAs at glevel 5) waited on
// its chain of exponentials: 0.225 ms at glevel 5, 40 levels.
constexpr int kRtWarps = 8;
__global__ void __launch_bounds__(32 * kRtWarps) rt_column_kernel(Geometry g, Phys P, RtConst c,
                                                                 RtFields f, State s) {
    extern __shared__ double lev_sm[]; // [4][nv][32]
    __shared__ double        s_cz[32], s_ins[32], s_up0[32], s_swtop[32], s_ptop[32];
    const int x = threadIdx.x, y = threadIdx.y;
    const int id = g.tile0 * 32 + blockIdx.x * 32 + x;
    const bool   valid = id < g.col_end;
    step_begin();
    step_wait();
    const RtStep st    = *f.step;
    const int    nv = g.nv, Np = g.Np, nvi = g.nvi;
    const double* Alt  = g.Altitude;
    const double* Alth = g.Altitudeh;
    const double  A = P.A, gravit = P.Gravit, ps0 = P.P_Ref, timestep = P.timestep;
    const double  lat = valid ? g.lat[id] : 0.0;
    const long long nstep = st.cur;
    if (y == 0 && valid) {
        // ---- calc_zenith + compute_cos_zenith_angles (insolation.cu:128-207) ----
        const double lon = g.lon[id];
        const bool   obl = !(c.obliquity < 1e-10);
        double       cz;
        if (c.sync_rot && c.ecc < 1e-10)
            cz = obl ? (sin(lat) * st.sin_decl + cos(lat) * st.cos_decl * cos(lon - c.alpha_i))
                     : cos(lat) * cos(lon - c.alpha_i);
        else if (c.sync_rot && !obl)
            cz = cos(lat) * cos(lon - st.alpha);
        else
            cz = (sin(lat) * st.sin_decl + cos(lat) * st.cos_decl * cos(lon - st.alpha));
        cz               = cz < 0.0 ? 0.0 : cz;
        f.cos_zenith[id] = cz;
        if (st.run) {
            const double coszrs = c.rt1Dmode ? 0.5 : cz;
            // insolation at the top (radcsw, profx_RT.h:74; 0 on the night side) and its first-orbit
            // average (annual_insol, profx_RT.h:30-37), for every column in either mode
            const double ins = coszrs > 0.0 ? c.incflx * pow(st.r_orb, -2) * coszrs : 0.0;
            f.insol[id]      = ins;
            if (nstep * timestep < (2 * M_PI / c.mean_motion))
                f.insol_ann[id] = f.insol_ann[id] * (nstep - 1) / nstep + ins / nstep;
            s_cz[x]  = coszrs;
            s_ins[x] = ins;
        }
    }
    if (!st.run) // uniform
        return;
    const bool on = valid && !(f.fallback && !(f.fallback[id] || recheck_column(id, f.period, nstep)));
    __syncthreads();
    const double coszrs = on ? s_cz[x] : 0.0;
    double *     sTr = lev_sm + x, *sEd = sTr + (size_t)nv * 32, *sEu = sEd + (size_t)nv * 32,
           *sSw = sEu + (size_t)nv * 32;
    auto P_ = [&](int lev) { return s.p[lev * Np + id]; };
    auto T_ = [&](int lev) { return s.T[lev * Np + id]; };
    const double bc = 5.677036E-8;
    auto         planck = [&](double t) { return bc * t * t * t * t; };
    const double* lt = g.lt;
    // interface temperatures (profx_RT.h:419-466)
    auto th_ = [&](int lev, double below, double above) { // T of the layers below and above
        return lev == 0 ? above
                        : lev == nv ? below : below * lt[kLtHIntt * nvi + lev] + above * lt[kLtHIntl * nvi + lev];
    };
    if (on) {
        const double kappa_lw_lat =
            c.latf_lw ? c.kappa_lw + (c.kappa_lw_pole - c.kappa_lw) * pow(sin(lat), 2) : c.kappa_lw;
        const double da = c.diff_ang;
        for (int lev = y; lev < nv; lev += kRtWarps) {
            const int    i  = lev * Np + id;
            const double p  = s.p[i], T = s.T[i], rho = s.Rho[i];
            const double pm = lev > 0 ? P_(lev - 1) : 0.0, Tm = lev > 0 ? T_(lev - 1) : T;
            const double Tp = lev < nv - 1 ? T_(lev + 1) : T;
            const double tb = th_(lev, Tm, T), tt = th_(lev + 1, T, Tp);
            double       ph;
            if (lev == 0) {
                const double psm = P_(1) - rho * gravit * (-Alt[0] - Alt[1]);
                ph               = 0.5 * (p + psm);
            }
            else
                ph = pm * lt[kLtHIntt * nvi + lev] + p * lt[kLtHIntl * nvi + lev];
            f.phtemp[i] = ph;
            f.thtemp[i] = tb;
            f.ttemp[i]  = T;
            if (lev == nv - 1) {
                double pp = pm + (p - pm) / (Alt[nv - 1] - Alt[nv - 2])
                                     * (2 * Alth[nv] - Alt[nv - 1] - Alt[nv - 2]);
                if (pp < 0)
                    pp = 0;
                s_ptop[x]        = 0.5 * (p + pp);
                f.phtemp[i + Np] = s_ptop[x];
                f.thtemp[i + Np] = T;
            }
            // computetau (profx_RT.h:278-314)
            const double dz = Alth[lev + 1] - Alth[lev];
            const double t0 = c.n_sw * c.kappa_sw * opacity_pow(p / ps0, c.n_sw - 1) * rho * dz;
            double       t1 = kappa_lw_lat
                        * (1 + c.n_lw * (1 - c.f_lw) / c.f_lw * opacity_pow(p / ps0, c.n_lw - 1))
                        * rho * dz;
            if (t1 < 0.0) // radclw's floor
                t1 = 0.0;
            f.tau[i]           = t0;
            f.tau[nv * Np + i] = t1;
            // the layer's transmissions and sources, downward and upward (radclw, profx_RT.h:162-275)
            const double bb = planck(tb), bl = planck(T), bt = planck(tt);
            const double ex = exp(-(t1 / 2.0) / da);
            if (t1 >= 1e-10) {
                const double q = da / (t1 / 2.0);
                sEd[lev * 32]  = source_func_lin(bb, bl, bt, q, ex);
                sEu[lev * 32]  = source_func_lin(bt, bl, bb, q, ex);
            }
            else {
                sEd[lev * 32] = source_thin(bb, bl, bt, (t1 / 2.0) / da, ex);
                sEu[lev * 32] = source_thin(bt, bl, bb, (t1 / 2.0) / da, ex);
            }
            sTr[lev * 32] = exp(-(1. / da) * t1);
            sSw[lev * 32] = coszrs > 0.0 ? exp(-(1.0 / coszrs) * t0) : 0.0;
        }
    }
    __syncthreads();
    if (on && y == 0) { // longwave down, then up from the reflecting lower boundary
        double dn = 0.0;
        for (int lev = nv - 1; lev >= 0; lev--) {
            dn            = sEd[lev * 32] + dn * sTr[lev * 32];
            sEd[lev * 32] = dn;
        }
        double up = bc * c.Tint * c.Tint * c.Tint * c.Tint;
        up += dn;
        s_up0[x] = up;
        for (int lev = 0; lev < nv; lev++) {
            up            = sEu[lev * 32] + up * sTr[lev * 32];
            sEu[lev * 32] = up; // at interface lev + 1
        }
    }
    else if (on && y == 1) { // shortwave down (radcsw, profx_RT.h:39-118)
        double sw = 0.0;
        if (coszrs > 0.0) {
            const double tau = (c.kappa_sw / gravit) * s_ptop[x];
            sw               = s_ins[x] * (1.0 - c.albedo) * exp(-(1.0 / coszrs) * tau);
        }
        s_swtop[x] = sw;
        for (int lev = nv - 1; lev >= 0; lev--) {
            sw            = sw * sSw[lev * 32];
            sSw[lev * 32] = sw; // at interface lev
        }
    }
    __syncthreads();
    if (!on)
        return;
    if (y == 0) {
        const double rscale = P.DeepModel ? (A + Alth[nv]) / A : 1.0;
        const int    t      = nv * Np + id;
        f.ASR[id]   = s_swtop[x] * g.areasT[id] * pow(rscale, 2);
        f.OLR[id]   = sEu[(nv - 1) * 32] * g.areasT[id] * pow(rscale, 2);
        f.fsw_up[t] = 0.0;
        f.fsw_dn[t] = s_swtop[x];
        f.flw_up[t] = sEu[(nv - 1) * 32];
        f.flw_dn[t] = 0.0;
    }
    for (int lev = y; lev < nv; lev += kRtWarps) {
        const int    i   = lev * Np + id;
        const double swl = sSw[lev * 32], swh = lev == nv - 1 ? s_swtop[x] : sSw[(lev + 1) * 32];
        const double dnl = sEd[lev * 32], dnh = lev == nv - 1 ? 0.0 : sEd[(lev + 1) * 32];
        const double upl = lev == 0 ? s_up0[x] : sEu[(lev - 1) * 32], uph = sEu[lev * 32];
        f.fsw_up[i] = 0.0;
        f.fsw_dn[i] = swl;
        f.flw_up[i] = upl;
        f.flw_dn[i] = dnl;
        const double dzr = Alth[lev] - Alth[lev + 1];
        double       d   = 0.0;
        if (coszrs > 0.0)
            d = -((0.0 - swl) - (0.0 - swh)) / dzr;
        d = d - ((upl - dnl) - (uph - dnh)) / dzr;
        if (!f.fallback) { // in surrogate mode the combine kernel limits and couples
            // cooling limiter and coupling to the dynamical core (profx_RT.h:560-584)
            const double p = s.p[i];
            if (p + s.Rd[i] / (s.Cp[i] - s.Rd[i]) * d * timestep < 0)
                d = -p / timestep;
            f.qheat[i] = d;
            s.Qheat[i] += st.Qheat_scaling * d;
        }
        f.dtemp[i] = d;
    }
}

} // namespace

void launch_rt(const Geometry& g, const Phys& P, const RtConst& c, const RtFields& f,
               const State& s, cudaStream_t st) {
    launch_step(rt_orbit_kernel, 1, 1, 0, st, c, P, f.step);
    const size_t     smem = sizeof(double) * 4 * 32 * g.nv;
    static SmemOptIn opt;
    if (opt.ensure(rt_column_kernel, smem) == cudaSuccess)
        launch_step(rt_column_kernel, g.ntile, dim3(32, kRtWarps), smem, st, g, P, c, f, s);
}

} // namespace thorx
