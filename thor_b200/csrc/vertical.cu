// The vertically implicit part of the small steps:
//   Prepare_Implicit_Vertical / _Poles (src/headers/dyn/thor_vertical_int.h:566-771),
//   Vertical_Eq (:52-563, the Thomas elimination and back substitution, FP64),
//   Density_Pressure_Eqs / _Poles (src/headers/dyn/thor_fastmodes.h:255-847).
//
// Split by what changes when. Once per RK stage (flux_kernel, stage_kernel): everything the
// stage's 1, 3 or 6 small steps share. The tridiagonal rows a, b, c depend on the stage's enthalpy
// and effective gravity only, so the elimination's divisions are done once and kept as factors
// (t = 1 / (b - c' a), vinv = CRdd t, va = a t, vc = c'); what is left of a small step's solve is one
// multiply-add per interface in each direction. The flux of the stage's own momentum Mhk, Whk is
// linear and constant, so its divergence (vdiv) is added instead of gathered again. Per small step:
// flux_kernel, the horizontal divergences of Mhs, h Mhs and pt Mhs (a plane kernel: 5 gathered
// fields instead of the 8 with Mhk), and column_kernel, the solve and the update.
//
// glevel 6, 48 levels, one B200, per small step: flux 55 us (3.4 TB/s of its 12 cell planes), column 69
// us (4 TB/s of its 17), and the stage's planes 164 us three times a step (with the vertical part of the
// slow modes); the fused kernel this replaces took 227 us per small step (three lockstep waves of CTAs,
// each phase waiting on its own loads; 26 cell planes of traffic).
#include "dyn_common.cuh"
#include "planes.cuh"

namespace thorx {
namespace {

constexpr int kTile  = kTileCols;
constexpr int kWarps = 8; // warps of a column CTA, each a contiguous chunk of levels

// (1 + s)^a - 1 for |s| <= 1/32 and 0 < a <= 4: the binomial series as a nested product, its eleventh
// term on below 2^-57 of the first (the binomial theorem; no cancellation, so the result is good to
// a few units in its own last place, where pow(1 + s, a) - 1 would keep only those of 1).
constexpr double kSeriesMax = 1.0 / 32.0;
__device__ __forceinline__ double pow1m(double s, double a) {
    const double b = a + 1.0;
    double       t = 1.0;
#pragma unroll
    for (int n = 10; n >= 1; n--) // coefficient (a - n) / (n + 1)
        t = fma(s * fma(b, 1.0 / (n + 1), -1.0), t, 1.0);
    return a * s * t;
}

// The entropy form's new pressure deviation in general (thor_fastmodes.h:255-847): P_Ref (Rd (F +
// (P_Ref / Rd) (p / P_Ref)^(Cv/Cp)) / P_Ref)^(Cp/Cv) - pk, F the increment of rho times the potential
// temperature. Called where the series does not hold (deviations above 1/32 of the pressure).
__device__ __noinline__ double pressure_general(double ps, double pk, double F, double Rd, double Cp,
                                                double P_Ref) {
    const double Cv = Cp - Rd;
    const double u  = P_Ref / Rd * pow((ps + pk) / P_Ref, Cv / Cp);
    return P_Ref * pow(Rd * (F + u) / P_Ref, Cp / Cv) - pk;
}

// ---------------------------------------------------------------------------------------------
// Horizontal divergences of a small step (and of a stage). Per column the 21 weights of div stay in
// registers; f_j = div_j . M_j is formed once per point and serves every flux. What bounds it: the
// bytes (12 cell planes for kSmall) and the 35 shared-memory reads a cell needs.
//   kSmall: Mhs, h, cen (pt or h + ep + ek), ps, Rhos, Slowp, SlowRho -> fx = ps + dt Sp,
//           fy = Rhos + dt Sd, ff = div(Mhs cen), Sp and Sd of Prepare_Implicit_Vertical
//   else:   Mhk, h, cen -> SlowRho = div(Mhk), Slowp = div(Mhk h), vdiv = div(Mhk cen), which
//           stage_kernel completes (slow false: vdiv only)
// ---------------------------------------------------------------------------------------------
// The ring's levels: what fits shared memory beside the halo (two CTAs an SM for rhombi).
template<int PITCH>
constexpr int kFluxStages = PITCH == kPitchRhombus ? 4 : PITCH == kPitchAny ? 3 : 2;
template<bool kSmall, bool kUni, int PITCH>
__global__ void __launch_bounds__(kPlaneCols, PITCH == kPitchRhombus ? 2 : 1)
    flux_kernel(Geometry g, Phys P, State s, double dt, bool slow) {
    constexpr int NG = 5, NO = kSmall ? 4 : 0;
    constexpr int kStages = kFluxStages<PITCH>;
    extern __shared__ __align__(16) double ring[];
    const int     Np = g.Np, nv = g.nv, nvi = g.nvi;
    const size_t  plane = (size_t)nv * Np;
    const double* M     = kSmall ? s.Mhs : s.Mhk;
    const double* cen   = P.energy ? s.cen : s.pt;
    double        d[7][3];
    int           pt[7];
    auto          seg = [&](const PlaneTile& t) {
        const bool valid = t.c < g.N;
#pragma unroll
        for (int j = 0; j < 7; j++) {
            pt[j] = t.point(j);
            const bool use = valid && (j == 0 || pt[j] != t.own); // not a hole
#pragma unroll
            for (int k = 0; k < 3; k++)
                d[j][k] = use ? __ldg(g.div + (size_t)(j * 3 + k) * Np + t.c) : 0.0;
        }
    };
    auto comp = [&](const PlaneTile& t, const double* b, int lev) {
        double F = 0.0, Fh = 0.0, Fc = 0.0;
#pragma unroll
        for (int j = 0; j < 7; j++) {
            const double* q = b + pt[j];
            const double  f = fma(d[j][2], q[2 * PITCH], fma(d[j][1], q[PITCH], d[j][0] * q[0]));
            F  = F + f;
            Fh = fma(f, q[3 * PITCH], Fh);
            Fc = fma(f, q[4 * PITCH], Fc);
        }
        if (!t.store)
            return;
        const int    c = t.c, i = lev * Np + c;
        const double rscale = g.lt[kLtRscale * nvi + lev];
        if constexpr (kSmall) {
            const double* o   = b + NG * PITCH + threadIdx.x;
            const double  RoC = rd_at<kUni>(P, s, i) / (cp_at<kUni>(P, s, i) - rd_at<kUni>(P, s, i));
            const double  Sp  = o[2 * kPlaneCols] - RoC * (rscale * Fh);
            const double  Sd  = o[3 * kPlaneCols] - rscale * F;
            s.fx[i] = fma(dt, Sp, o[0]);
            s.fy[i] = fma(dt, Sd, o[kPlaneCols]);
            s.ff[i] = rscale * Fc;
        }
        else {
            s.vdiv[i] = rscale * Fc;
            if (slow) {
                s.SlowRho[i] = rscale * F;
                s.Slowp[i]   = rscale * Fh;
            }
        }
    };
    if constexpr (kSmall) {
        const double* const src[NG + NO] = {M,    M + plane, M + 2 * plane, s.h, cen,
                                            s.ps, s.Rhos,    s.Slowp,       s.SlowRho};
        plane_loop<NG, NO, PITCH, kStages>(g, ring, src, seg, comp);
    }
    else {
        const double* const src[NG + NO] = {M, M + plane, M + 2 * plane, s.h, cen};
        plane_loop<NG, NO, PITCH, kStages>(g, ring, src, seg, comp);
    }
}

// ---------------------------------------------------------------------------------------------
// Thermodynamics of an RK stage (Compute_Temperature_H_Pt_Geff, src/headers/dyn/thor_auxiliary.h:55-309,
// calcT = true): T, enthalpy, potential temperature (or the energy form's energies) at the centres,
// their interface values, the effective gravity. A CTA is a tile of 32 columns; a warp walks a
// contiguous chunk of levels upward and carries the level below, so that each level's potential
// temperature costs one pow (one more per chunk), where the level-strided form evaluated two.
// ---------------------------------------------------------------------------------------------
template<bool kUni>
__global__ void __launch_bounds__(kTile* kWarps, 3) thermo_kernel(Geometry g, Phys P, State s) {
    const int nv = g.nv, nvi = g.nvi, Np = g.Np;
    const int c  = (g.tile0 + blockIdx.x) * kTile + threadIdx.x;
    const int chunk = (nv + kWarps - 1) / kWarps;
    const int l0 = threadIdx.y * chunk, l1 = min(nv, l0 + chunk);
    step_begin();
    step_wait();
    if (c >= g.N || l0 >= l1)
        return;
    const double* Alt  = g.Altitude;
    const double* Alth = g.Altitudeh;
    const double* lt   = g.lt;
    const double  A = P.A, P_Ref = P.P_Ref, Gravit = P.Gravit;
    const bool    eeq = P.energy, ghv = P.GravHeightVar;
    const size_t  plane = (size_t)nv * Np;
    struct Level {
        double p, rho, Rd, Cp, h, pt, ep, ek; // pt: entropy form; ep, ek: energy form
    };
    auto state = [&](int lev) {
        const int i = lev * Np + c;
        Level     q{};
        q.p   = s.pk[i];
        q.rho = s.Rhok[i];
        q.Rd  = rd_at<kUni>(P, s, i);
        q.Cp  = cp_at<kUni>(P, s, i);
        return q;
    };
    auto derive = [&](Level& q, int lev) { // returns T (thor_auxiliary.h:111-163)
        const double Cv = q.Cp - q.Rd, T = q.p / (q.rho * q.Rd);
        q.h = Cv * T + q.p / q.rho;
        if (eeq) {
            const int    i  = lev * Np + c;
            const double m0 = s.Mhk[i], m1 = s.Mhk[plane + i], m2 = s.Mhk[2 * plane + i], w = s.Wk[i];
            q.ep = ghv ? Gravit * lt[kLtGhv * nvi + lev] * Alt[lev] : Gravit * Alt[lev];
            q.ek = 0.5 * (m0 * m0 + m1 * m1 + m2 * m2 + w * w) / (q.rho * q.rho);
        }
        else
            q.pt = (P_Ref / (q.Rd * q.rho)) * pow(q.p / P_Ref, Cv / q.Cp);
        return T;
    };
    // velocity-weighted effective gravity at interior interface i (:288-289)
    auto gravity = [&](int i, double rhoh, double dp_dz) {
        return -(s.Whk[i * Np + c] / rhoh) * dp_dz;
    };
    Level  lo{};
    double gw = 0.0; // gravity at the interface below the current level
    if (l0 > 0) {
        lo = state(l0 - 1);
        derive(lo, l0 - 1);
    }
    for (int lev = l0; lev < l1; lev++) {
        const int    i   = lev * Np + c;
        const double alt = Alt[lev];
        Level        q   = state(lev);
        const double T   = derive(q, lev);
        s.T[i]           = T;
        s.h[i]           = q.h;
        if (eeq) {
            s.ep[i]     = q.ep;
            s.ek[i]     = q.ek;
            s.Etotal[i] = q.rho * (q.ep + q.ek) + (q.Cp - q.Rd) / q.Rd * q.p;
            s.cen[i]    = q.h + q.ep + q.ek;
        }
        else
            s.pt[i] = q.pt;
        if (lev > 0) { // interior interface `lev`
            const double intt = lt[kLtHIntt * nvi + lev], intl = lt[kLtHIntl * nvi + lev];
            const double dp_dz = (q.p - lo.p) / (alt - Alt[lev - 1]);
            const double rhoh  = lo.rho * intt + q.rho * intl;
            const double hh    = lo.h * intt + q.h * intl;
            s.hh[i]            = hh;
            if (eeq) {
                const double eph = lo.ep * intt + q.ep * intl, ekh = lo.ek * intt + q.ek * intl;
                s.eph[i]  = eph;
                s.ekh[i]  = ekh;
                s.face[i] = hh + eph + ekh;
            }
            else
                s.pth[i] = lo.pt * intt + q.pt * intl;
            s.gtilh[i]      = -(1.0 / rhoh) * dp_dz;
            const double gu = gravity(lev, rhoh, dp_dz);
            // effective gravity at the centre of the level below (:293-300)
            if (lev > l0)
                s.gtil[i - Np] = gw * lt[kLtCIntt * nvi + lev] + gu * lt[kLtCIntl * nvi + lev];
            gw = gu;
        }
        else { // bottom boundary, extrapolated (:167-187)
            const Level  up   = state(1);
            const double extr = (-alt - Alt[1]) / (Alt[1] - alt);
            s.hh[c]           = q.h;
            const double gr   = ghv ? Gravit * pow(A / (A + Alt[0]), 2) : Gravit;
            const double pl   = up.p - q.rho * gr * (-alt - Alt[1]);
            const double rhol = up.rho + (up.rho - q.rho) * extr;
            const double rhoh = 0.5 * (q.rho + rhol);
            s.gtilh[c]        = -(1.0 / rhoh) * ((q.p - pl) / (2.0 * Alt[0]));
        }
        if (lev == 1) { // extrapolations to the bottom interface from levels 0 and 1 (:188-258)
            const double e = (Alth[0] - Alt[1]) / (Alt[1] - Alt[0]);
            if (eeq) {
                const double eph = ghv ? Gravit * pow(A / (A + Alth[0]), 2) * Alth[0] : Gravit * Alth[0];
                const double ekh = q.ek + (q.ek - lo.ek) * e;
                s.eph[c]  = eph;
                s.ekh[c]  = ekh;
                s.face[c] = lo.h + eph + ekh;
            }
            else
                s.pth[c] = q.pt + (q.pt - lo.pt) * e;
        }
        if (lev == nv - 1) { // top boundary (:188-266)
            const int    it   = nv * Np + c;
            const double far  = 2 * Alth[nv] - alt - Alt[nv - 2];
            const double extr = far / (Alt[nv - 1] - Alt[nv - 2]);
            s.hh[it]          = q.h;
            const double rhop = lo.rho + (q.rho - lo.rho) * extr;
            const double rhoh = 0.5 * (q.rho + rhop);
            if (eeq) {
                const double eph =
                    ghv ? Gravit * pow(A / (A + Alth[nv]), 2) * Alth[nv] : Gravit * Alth[nv];
                const double ekh = lo.ek + (q.ek - lo.ek) * extr;
                s.eph[it]  = eph;
                s.ekh[it]  = ekh;
                s.face[it] = q.h + eph + ekh;
            }
            else
                s.pth[it] = lo.pt + (q.pt - lo.pt) * extr;
            const double gr = ghv ? Gravit * pow(A / (A + Alt[nv - 1]), 2) : Gravit;
            const double pp = lo.p - q.rho * gr * far;
            s.gtilh[it]     = -(1.0 / rhoh) * ((pp - q.p) / (2.0 * (Alth[nv] - Alt[nv - 1])));
            // the reference interpolates with the top layer's own geometry, 0 above (:259-266)
            s.gtil[i] = gw * lt[kLtCIntt * nvi + lev] + 0.0 * lt[kLtCIntl * nvi + lev];
        }
        lo = q;
    }
    if (l1 < nv) { // the chunk's last centre needs the gravity at the next chunk's lower interface
        const Level  q = state(l1);
        const double intt = lt[kLtHIntt * nvi + l1], intl = lt[kLtHIntl * nvi + l1];
        const double gu = gravity(l1, lo.rho * intt + q.rho * intl,
                                  (q.p - lo.p) / (Alt[l1] - Alt[l1 - 1]));
        s.gtil[(l1 - 1) * Np + c] = gw * lt[kLtCIntt * nvi + l1] + gu * lt[kLtCIntl * nvi + l1];
    }
}

// ---------------------------------------------------------------------------------------------
// What a stage's small steps share, by column: the slow modes' vertical parts (slow; Compute_Slow_Modes,
// src/headers/dyn/thor_slowmodes.h:48-683, the horizontal divergences and the work of the pressure
// gradient already in place), the stage's own flux and sources, and the rows of Vertical_Eq with their
// elimination (thor_vertical_int.h:188-484). Levels in parallel; the rows in shared memory, where one warp
// runs the chain of dependent divisions. vc is 0 at the top row.
// ---------------------------------------------------------------------------------------------
template<bool kUni>
__device__ __forceinline__ double crdd_of(const Geometry& g, const Phys& P, const State& s, int c,
                                          int lev, double deltat) {
    const int    iu = lev * g.Np + c, il = iu - g.Np;
    const double Rl = rd_at<kUni>(P, s, il), Ru = rd_at<kUni>(P, s, iu);
    const double CRddl = (cp_at<kUni>(P, s, il) - Rl) / (Rl * deltat * deltat);
    const double CRddu = (cp_at<kUni>(P, s, iu) - Ru) / (Ru * deltat * deltat);
    const double alth = g.Altitudeh[lev], alt = g.Altitude[lev], altl = g.Altitude[lev - 1];
    return div_rcp(CRddl * (alt - alth) + CRddu * (alth - altl), alt - altl,
                   g.lt[kLtDzh * g.nvi + lev]);
}

template<bool kUni>
__global__ void __launch_bounds__(kTile* kWarps, 3) stage_kernel(Geometry g, Phys P, State s,
                                                                 double deltat, bool keep, bool slow) {
    extern __shared__ double rows[]; // a, b, c: [3][nv][32]
    const int  nv = g.nv, nvi = g.nvi, Np = g.Np, x = threadIdx.x;
    const int  c      = (g.tile0 + blockIdx.x) * kTile + x;
    const bool active = c < g.N;
    double *   sa = rows + x, *sb = sa + (size_t)nv * kTile, *sc = sb + (size_t)nv * kTile;
    const double* Alt  = g.Altitude;
    const double* Alth = g.Altitudeh;
    const double* lt   = g.lt;
    const double  Gravit = P.Gravit;
    const bool    deep = P.DeepModel, nonh = P.NonHydro, ghv = P.GravHeightVar;
    const double* face = P.energy ? s.face : s.pth;
    const bool    pole = active && (g.cflag[c] & kPole) != 0;
    step_begin();
    step_wait();
    if (active)
        for (int lev = threadIdx.y; lev < nv; lev += kWarps) {
            const int    i  = lev * Np + c;
            const double whl = lev == 0 ? 0.0 : s.Whk[i], wht = s.Whk[i + Np];
            const double fcl = face[i], fct = face[i + Np];
            const double Rd = rd_at<kUni>(P, s, i), Cv = cp_at<kUni>(P, s, i) - Rd;
            const double dpr = s.diffpr[i], qh = s.Qheat[i], rho = s.Rhok[i];
            double       r2p = 1.0, r2l = 1.0;
            if (deep) {
                r2p = lt[kLtR2hD * nvi + lev + 1];
                r2l = lt[kLtR2hD * nvi + lev];
            }
            const double rdz    = lt[(deep ? kLtRDzR2m : kLtRDz) * nvi + lev];
            const double rthick = deep && !pole ? lt[kLtRDr2dz * nvi + lev] : rdz;
            const double wt = wht * r2p, wl = whl * r2l;
            s.vdiv[i] = fma(fma(wt, fct, -(wl * fcl)), rdz, s.vdiv[i]);
            if (P.energy)
                s.vsrc[i] = dpr + qh;
            else {
                s.vsrc[i] = fma(Rd / Cv, qh, dpr);
                s.vru[i]  = 1.0 / (s.pt[i] * rho);
            }
            if (slow) {
                const double dwdz  = (wt - wl) * rthick;
                const double dwhdz = (wt * s.hh[i + Np] - wl * s.hh[i]) * rdz;
                s.SlowRho[i]       = -(s.SlowRho[i] + dwdz) + s.diffrh[i];
                const double q     = Rd / Cv * (-s.Slowp[i] - s.gtil[i] - dwhdz + s.fx[i] + qh);
                s.Slowp[i]         = q + (P.energy ? Rd / Cv * dpr : dpr);
                double sw          = 0.0;
                if (lev > 0) { // the slow vertical tendency at the lower interface
                    const int    il = i - Np;
                    const double intt = lt[kLtHIntt * nvi + lev], intl = lt[kLtHIntl * nvi + lev];
                    double       gl = Gravit, gu = Gravit;
                    if (ghv) {
                        gl *= lt[kLtGhv * nvi + lev - 1];
                        gu *= lt[kLtGhv * nvi + lev];
                    }
                    double lo = s.Rhok[il] * gl, up = rho * gu;
                    if (deep) {
                        lo += s.fy[il];
                        up += s.fy[i];
                    }
                    double swr = lo * intt + up * intl;
                    if (nonh)
                        swr -= s.diffw[il] * intt + s.diffw[i] * intl;
                    swr += (s.pk[i] - s.pk[il]) / (Alt[lev] - Alt[lev - 1]);
                    if (P.drag)
                        swr -= s.dWh[i];
                    sw = -swr;
                }
                s.SlowWh[i] = sw;
                if (lev == nv - 1)
                    s.SlowWh[i + Np] = 0.0;
            }
            if (lev == 0)
                continue;
            const double alth = Alth[lev], alt = Alt[lev], altl = Alt[lev - 1];
            double       hp = s.hh[(lev + 1) * Np + c], h = s.hh[lev * Np + c], hm = s.hh[(lev - 1) * Np + c];
            const double gp = s.gtilh[(lev + 1) * Np + c], gg = s.gtilh[lev * Np + c], gm = s.gtilh[(lev - 1) * Np + c];
            const int    il = i - Np;
            const double Rl = rd_at<kUni>(P, s, il), Ru = Rd;
            const double Cl = cp_at<kUni>(P, s, il) - Rl, Cu = Cv;
            double       GCoRl, GCoRu;
            if (ghv) {
                GCoRl = Gravit * lt[kLtGhv * nvi + lev - 1] * Cl / Rl;
                GCoRu = Gravit * lt[kLtGhv * nvi + lev] * Cu / Ru;
            }
            else {
                GCoRl = Gravit * Cl / Rl;
                GCoRu = Gravit * Cu / Ru;
            }
            const double dzp   = lt[kLtDzp * nvi + lev];
            const double dzh   = lt[kLtDzh * nvi + lev]; // RN(1 / (alt - altl))
            const double dzm   = lt[kLtDzm * nvi + lev];
            const double dzph  = dzp * dzh;
            const double dzmh  = dzm * dzh;
            const double intl  = lt[kLtIntl * nvi + lev];
            const double inttm = lt[kLtInttm * nvi + lev];
            const double CRdd  = nonh ? crdd_of<kUni>(g, P, s, c, lev, deltat) : 0.0;
            const double GCoR  = div_rcp(GCoRl * (alt - alth) + GCoRu * (alth - altl), alt - altl, dzh);
            double       aa, bb, cc;
            if (deep) {
                hp                = hp * lt[kLtR2hI * nvi + lev + 1];
                h                 = h * lt[kLtR2hI * nvi + lev];
                hm                = hm * lt[kLtR2hI * nvi + lev - 1];
                const double or2  = lt[kLtOr2 * nvi + lev];
                const double tor3 = lt[kLtTor3 * nvi + lev];
                cc                = -dzph * or2 * hp - inttm * (gp + GCoR - tor3 * hp);
                bb = (dzph + dzmh) * or2 * h + (intl - inttm) * (gg + GCoR - tor3 * h);
                aa = -dzmh * or2 * hm + intl * (gm + GCoR - tor3 * hm);
            }
            else {
                cc = -dzph * hp - inttm * (gp + GCoR);
                bb = (dzph + dzmh) * h + (intl - inttm) * (gg + GCoR);
                aa = -dzmh * hm + intl * (gm + GCoR);
            }
            if (nonh)
                bb += CRdd;
            sa[lev * kTile] = aa;
            sb[lev * kTile] = bb;
            sc[lev * kTile] = cc;
            if (keep) {
                s.vrows[(size_t)lev * Np + c]                         = aa;
                s.vrows[(size_t)(nvi + lev) * Np + c]                 = bb;
                s.vrows[(size_t)(2 * nvi + lev) * Np + c]             = cc;
            }
        }
    __syncthreads();
    if (threadIdx.y == 0) {
        double cprev = 0.0;
#pragma unroll 4
        for (int lev = 1; lev < nv; lev++) { // lev 1: c' = c / b (its row has no lower neighbour)
            const double t  = 1.0 / (sb[lev * kTile] - cprev * sa[lev * kTile]);
            cprev           = sc[lev * kTile] * t;
            sb[lev * kTile] = t;
            sc[lev * kTile] = cprev;
        }
    }
    __syncthreads();
    if (active)
        for (int lev = 1 + threadIdx.y; lev < nv; lev += kWarps) {
            const double t = sb[lev * kTile];
            // the right-hand side carries the factor CRdd (:421-461)
            s.vinv[(size_t)lev * Np + c] = crdd_of<kUni>(g, P, s, c, lev, deltat) * t;
            s.va[(size_t)lev * Np + c]   = lev == 1 ? 0.0 : sa[lev * kTile] * t;
            s.vc[(size_t)lev * Np + c]   = lev == nv - 1 ? 0.0 : sc[lev * kTile];
        }
}

// ---------------------------------------------------------------------------------------------
// The solve and the update of one small step. A CTA is a tile of 32 columns; warp y owns the levels
// [y chunk, (y + 1) chunk) and the rows at their lower interfaces. With the stage's factors both
// sweeps are first-order linear recurrences, d'_l = e_l - va_l d'_(l-1) and w_l = d'_l - vc_l w_(l+1):
// each warp runs its chunk from a zero start and keeps the end value and the product of the
// coefficients, the warps' starts follow from these over shared memory, and a second pass from the
// true start gives the serial algorithm's values (one rounding apart in the start). So every warp
// streams its own planes and no warp waits for a sweep of the whole column. What bounds it: bytes,
// 17 cell planes.
// part: 0 all; 1 the solve only (Whs written); 2 the update only, with the Whs found in memory.
// ---------------------------------------------------------------------------------------------
// CTAs per SM and levels unrolled, chosen at glevel 6 by the launch alone: three CTAs of 80 registers with
// three levels' loads in flight 72.5 us; four CTAs of 64 registers 76.6 (two levels), 75.3 (three), 81.4
// (six); three CTAs 74.8 (two), 77.1 (six); with the next chunk's planes prefetched into L2 82. In the step
// with dependent launch, where the last wave of a launch overlaps the next one, us per Held-Suarez step at
// glevel 4 / 5 / 6 / 7 (32, 40, 48, 48 levels): three CTAs, three levels 474 / 1074 / 4236 / 17543; two
// levels 472 / 1073 / 4237 / 17566; six 483 / 1086 / 4260 / 17596; two CTAs, three levels 464 / 1190 / 4468 /
// 18190; four CTAs, two levels 484 / 1063 / 4165 / 16890; three levels 495 / 1086 / 4246 / 17085. Four CTAs
// with two levels would be the better choice from glevel 5 on, by 1 to 4 %, and the worse one at glevel 4.
constexpr int kColOcc = 3, kColUnroll = 3;
template<bool kUni>
__global__ void __launch_bounds__(kTile* kWarps, kColOcc)
    column_kernel(Geometry g, Phys P, State s, double deltat, int part, bool keep) {
    extern __shared__ double sd[]; // e, then d': [nv][32]
    __shared__ double        t_end[kWarps][kTile], t_mul[kWarps][kTile];
    __shared__ double        u_end[kWarps][kTile], u_mul[kWarps][kTile];
    const int  nv = g.nv, nvi = g.nvi, Np = g.Np, x = threadIdx.x, y = threadIdx.y;
    const int  c      = (g.tile0 + blockIdx.x) * kTile + x;
    const bool active = c < g.N;
    const int  chunk  = (nv + kWarps - 1) / kWarps;
    const int  l0 = min(nv, y * chunk), l1 = min(nv, l0 + chunk);
    double*    d = sd + x;
    const double* lt   = g.lt;
    const double  Gravit = P.Gravit;
    const bool    nonh = P.NonHydro, ghv = P.GravHeightVar, deep = P.DeepModel, eeq = P.energy;
    const bool    pole = active && (g.cflag[c] & kPole) != 0;
    double        wtop = 0.0; // the solution at interface l1
    step_begin();
    step_wait();
    if (part != 2) {
        // the rows' right-hand sides, scaled, and the elimination from a zero start
        double te = 0.0, tm = 1.0;
        if (active && l0 < l1) {
            const int r0 = max(l0, 1);
            double    X = s.fx[(r0 - 1) * Np + c], Y = s.fy[(r0 - 1) * Np + c];
#pragma unroll kColUnroll
            for (int lev = r0; lev < l1; lev++) {
                const int    i  = lev * Np + c;
                const double Xu = s.fx[i], Yu = s.fy[i];
                const double Srh = s.SlowWh[i], whs = nonh ? s.Whs[i] : 0.0;
                const double inv = s.vinv[i], a = s.va[i];
                const double dzh = lt[kLtDzh * nvi + lev];
                const double gl  = ghv ? Gravit * lt[kLtGhv * nvi + lev] : Gravit;
                const double Yh  = Y * lt[kLtHIntt * nvi + lev] + Yu * lt[kLtHIntl * nvi + lev];
                const double rhs = whs - deltat * ((Xu - X) * dzh + gl * Yh - Srh);
                if (keep)
                    s.vrows[(size_t)(3 * nvi + lev) * Np + c] =
                        crdd_of<kUni>(g, P, s, c, lev, deltat) * rhs;
                const double e = rhs * inv;
                d[lev * kTile] = e;
                te             = fma(-a, te, e);
                tm             = -a * tm;
                X              = Xu;
                Y              = Yu;
            }
        }
        t_end[y][x] = te;
        t_mul[y][x] = tm;
        __syncthreads();
        // the true start, d' over e, and the back substitution from a zero start
        double ue = 0.0, um = 1.0;
        if (active && l0 < l1) {
            double dp = 0.0;
            for (int k = 0; k < y; k++)
                dp = fma(t_mul[k][x], dp, t_end[k][x]);
            const int r0 = max(l0, 1);
#pragma unroll kColUnroll
            for (int lev = r0; lev < l1; lev++) {
                dp             = fma(-s.va[lev * Np + c], dp, d[lev * kTile]);
                d[lev * kTile] = dp;
            }
#pragma unroll kColUnroll
            for (int lev = l1 - 1; lev >= r0; lev--) {
                const double cc = s.vc[lev * Np + c];
                ue              = fma(-cc, ue, d[lev * kTile]);
                um              = -cc * um;
            }
        }
        u_end[y][x] = ue;
        u_mul[y][x] = um;
        __syncthreads();
        for (int k = kWarps - 1; k > y; k--)
            wtop = fma(u_mul[k][x], wtop, u_end[k][x]);
    }
    if (!active || l0 >= l1)
        return;
    const double* Alt  = g.Altitude;
    const double* Alth = g.Altitudeh;
    const double* face = eeq ? s.face : s.pth;
    if (part == 2)
        wtop = s.Whs[l1 * Np + c];
    else if (l1 == nv) {
        s.Whs[nv * Np + c] = 0.0;
        s.Whs[c]           = 0.0;
    }
    double wht = wtop, pht = part == 1 ? 0.0 : face[l1 * Np + c];
#pragma unroll kColUnroll
    for (int lev = l1 - 1; lev >= l0; lev--) {
        const int i   = lev * Np + c;
        double    whl = 0.0;
        if (lev > 0) {
            if (part == 2)
                whl = s.Whs[i];
            else {
                // the chunk's lowest value as the warp below composes it, so that both sides of the interface
                // (and a part-2 launch) see the same bits
                whl      = lev == l0 ? fma(u_mul[y][x], wtop, u_end[y][x])
                                     : fma(-s.vc[i], wht, d[lev * kTile]);
                s.Whs[i] = whl;
            }
        }
        if (part == 1) {
            wht = whl;
            continue;
        }
        // Density_Pressure_Eqs at this level
        const double Y = s.fy[i], F = s.ff[i], D = s.vdiv[i], src = s.vsrc[i], pk = s.pk[i];
        const double ph = face[i], ps = eeq ? 0.0 : s.ps[i], ru = eeq ? 0.0 : s.vru[i];
        double       r2p = 1.0, r2l = 1.0;
        if (deep) {
            r2p = lt[kLtR2hD * nvi + lev + 1];
            r2l = lt[kLtR2hD * nvi + lev];
        }
        const double rdzr2m = lt[(deep ? kLtRDzR2m : kLtRDz) * nvi + lev];
        const double rthick = deep && !pole ? lt[kLtRDr2dz * nvi + lev] : rdzr2m;
        const double phl = lev == 0 ? 0.0 : ph;
        const double dW  = fma(wht, r2p, -(whl * r2l));
        const double dWp = fma(wht * pht, r2p, -(whl * phl * r2l));
        const double rhos = fma(-(dW * rthick), deltat, Y);
        const double dF   = -(fma(dWp, rdzr2m, F) + D) * deltat;
        const double Rd = rd_at<kUni>(P, s, i), Cp = cp_at<kUni>(P, s, i), Cv = Cp - Rd;
        s.Rhos[i] = rhos;
        if (eeq) {
            const double aux = s.Etotal[i] + fma(src, deltat, dF);
            s.Etotal[i]      = aux;
            const size_t pl  = (size_t)nv * Np;
            const double m0 = s.Mhs[i] + s.Mhk[i], m1 = s.Mhs[pl + i] + s.Mhk[pl + i],
                         m2 = s.Mhs[2 * pl + i] + s.Mhk[2 * pl + i];
            const double whl2 = lev == 0 ? 0.0 : whl + s.Whk[i], wht2 = wht + s.Whk[i + Np];
            const double w = (whl2 * (Alth[lev + 1] - Alt[lev]) + wht2 * (Alt[lev] - Alth[lev]))
                             * lt[kLtRDz * nvi + lev];
            const double rho = rhos + s.Rhok[i];
            const double gz  = ghv ? Gravit * lt[kLtGhv * nvi + lev] * Alt[lev] : Gravit * Alt[lev];
            const double Epot_kin = rho * gz + 0.5 * (m0 * m0 + m1 * m1 + m2 * m2 + w * w) / rho;
            s.ps[i] = Rd / Cv * (aux - Epot_kin) - pk;
        }
        else {
            // relative to the stage's pressure: rho theta = U (1 + z), U = 1 / ru its value there
            const double sp = ps / pk;
            const double kap = Cv / Cp, ikap = Cp / Cv;
            const double z  = fma(dF, ru, pow1m(sp, kap));
            double       pn = pk * pow1m(z, ikap);
            if (!(fabs(sp) <= kSeriesMax && fabs(z) <= kSeriesMax && ikap <= 4.0))
                pn = pressure_general(ps, pk, dF, Rd, Cp, P.P_Ref);
            s.ps[i] = fma(src, deltat, pn);
        }
        wht = whl;
        pht = ph;
    }
}

template<bool kSmall, bool kUni, int PITCH>
void launch_flux_t(const Geometry& g, const Phys& P, const State& s, double dt, bool slow,
                   cudaStream_t st) {
    constexpr int    kStages = kFluxStages<PITCH>;
    constexpr size_t smem    = plane_ring_bytes<5, kSmall ? 4 : 0, PITCH, kStages>();
    static SmemOptIn opt;
    if (opt.ensure(flux_kernel<kSmall, kUni, PITCH>, smem) != cudaSuccess)
        return;
    const int per_sm = PITCH == kPitchRhombus ? 2 : 1;
    launch_step(flux_kernel<kSmall, kUni, PITCH>, plane_ctas(g, per_sm), kPlaneCols, smem, st, g, P, s, dt,
                slow);
}
// the layout of the grid's tiles (Geometry::rhombi, wide)
template<bool kSmall, bool kUni>
void launch_flux_u(const Geometry& g, const Phys& P, const State& s, double dt, bool slow,
                   cudaStream_t st) {
    if (g.rhombi)
        launch_flux_t<kSmall, kUni, kPitchRhombus>(g, P, s, dt, slow, st);
    else if (!g.wide)
        launch_flux_t<kSmall, kUni, kPitchAny>(g, P, s, dt, slow, st);
    else
        launch_flux_t<kSmall, kUni, kPitchWide>(g, P, s, dt, slow, st);
}

} // namespace

void launch_thermo(const Geometry& g, const Phys& P, const State& s, cudaStream_t st) {
    const dim3 block(kTile, kWarps);
    if (P.uniform_thermo)
        launch_step(thermo_kernel<true>, g.ntile, block, 0, st, g, P, s);
    else
        launch_step(thermo_kernel<false>, g.ntile, block, 0, st, g, P, s);
}

void launch_flux(const Geometry& g, const Phys& P, const State& s, double dt, cudaStream_t st) {
    if (P.uniform_thermo)
        launch_flux_u<true, true>(g, P, s, dt, false, st);
    else
        launch_flux_u<true, false>(g, P, s, dt, false, st);
}

void launch_stage(const Geometry& g, const Phys& P, const State& s, double dt, bool keep, bool slow,
                  cudaStream_t st) {
    launch_flux_u<false, true>(g, P, s, 0.0, slow, st);
    const size_t smem = sizeof(double) * 3 * g.nv * kTile;
    const dim3   block(kTile, kWarps);
    if (P.uniform_thermo) {
        static SmemOptIn opt;
        if (opt.ensure(stage_kernel<true>, smem) == cudaSuccess)
            launch_step(stage_kernel<true>, g.ntile, block, smem, st, g, P, s, dt, keep, slow);
    }
    else {
        static SmemOptIn opt;
        if (opt.ensure(stage_kernel<false>, smem) == cudaSuccess)
            launch_step(stage_kernel<false>, g.ntile, block, smem, st, g, P, s, dt, keep, slow);
    }
}

void launch_column(const Geometry& g, const Phys& P, const State& s, double dt, int part, bool keep,
                   cudaStream_t st) {
    const size_t smem = sizeof(double) * g.nv * kTile; // at most 32 KB (128 levels)
    const dim3   block(kTile, kWarps);
    if (P.uniform_thermo)
        launch_step(column_kernel<true>, g.ntile, block, smem, st, g, P, s, dt, part, keep);
    else
        launch_step(column_kernel<false>, g.ntile, block, smem, st, g, P, s, dt, part, keep);
}

} // namespace thorx
