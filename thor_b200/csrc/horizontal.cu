// Horizontal operators of the small steps as plane kernels (planes.cuh): the 3D divergence damping
// (DivM_Op / _Poles, src/headers/dyn/thor_div.h:49-535) and the horizontal momentum equation
// (Momentum_Eq / _Poles, src/headers/dyn/thor_fastmodes.h:54-253).
//
// The damping operator is the gradient of a divergence on the grid's triangles. The reference
// evaluates, per column, the divergence on its six (five) triangles and combines them along the
// cell's edges; a triangle is shared by three columns, so here its divergence D is computed once, by
// the column that owns it (two triangles per column: ring points 1, 2 and 2, 3), from 9 weights on the
// three vertices' momenta and 3 on their vertical momenta, and shared through shared memory; a tile's
// columns also need the triangles around its edge, which two more warps compute. Per cell that is 24
// multiply-adds for D and 18 for the gradient, all weights in registers, against 84 weights read from
// shared memory when the operator is applied to the stencil points directly. The terms are the
// reference's (its triangle sequence regrouped by vertex); the poles' triangles are kept apart, since
// the poles weigh the third corner's vertical momentum by the second sub-area (thor_div.h:443-454).
//
// Warps 0-7 hold the gradient's weights (thread = column), warps 8-15 the owned triangles' (thread =
// column); the gradient runs one level behind the triangles, so a level costs one barrier. 16 warps, so
// that every scheduler has four and a thread may hold 128 registers: with warps of their own for the edge
// triangles a scheduler had five and the weights spilled. The edge triangles go to the role with less to
// do (divm0: the gradient's warps; momentum: the triangle warps that copy no halo).
//
// glevel 6, 48 levels, one B200, us per launch, the column-tile form and this: divm0 91 and 53, momentum
// 109 and 59. divm0 by parts (timing copies; 62 us at that time): starting and the loop 11, own copies 7,
// halo copies 11, the edge triangles 13, the others 27; the bytes alone (7 planes) are 16 us. What bounds
// it is issue and the barrier a level costs: two levels per barrier need 200 registers and spill (62 -> 88
// us), the halo's copies spread over all warps cost more in index arithmetic than they balance.
#include "dyn_common.cuh"
#include "planes.cuh"

namespace thorx {
namespace {

constexpr int kDivThreads = 2 * kPlaneCols;
constexpr int PITCH = kPitchRhombus;

// ---- triangle and gradient weights (once per context) ------------------------------------------
struct TriGeo {
    const double *areas, *areasTr, *ti, *te, *oa;
    int           Np;
    __device__ double AR(int j, int v, int c) const { return areas[(size_t)(j * 3 + v) * Np + c]; }
    __device__ double AT(int j, int c) const { return areasTr[(size_t)j * Np + c]; }
    __device__ double TI(int j, int k, int c) const { return ti[(size_t)(j * 3 + k) * Np + c]; }
    __device__ double TE(int j, int k, int c) const { return te[(size_t)(j * 3 + k) * Np + c]; }
    __device__ double OA(int j, int k, int c) const { return oa[(size_t)(j * 3 + k) * Np + c]; }
    // triangle j of column c (of n): w[0..8] the vertices' vector weights (c, ring j, ring j + 1), w[9..11]
    // the weights of their vertical momentum
    __device__ void triangle(int c, int j, int n, bool pole, double* w) const {
        const int    q = (j + 1) % n;
        const double r = 0.5 / AT(j, c);
        for (int k = 0; k < 3; k++) {
            w[k]     = (TI(q, k, c) - TI(j, k, c)) * r;
            w[3 + k] = (TE(j, k, c) - TI(j, k, c)) * r;
            w[6 + k] = (TE(j, k, c) + TI(q, k, c)) * r;
        }
        for (int v = 0; v < 3; v++)
            w[9 + v] = AR(j, pole && v == 2 ? 1 : v, c) / AT(j, c);
    }
};

__global__ void tri_weights_kernel(Geometry g, double* tw, double* gw) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x, Np = g.Np;
    if (c >= g.N)
        return;
    const TriGeo t{g.areas, g.areasTr, g.nvecti, g.nvecte, g.nvecoa, Np};
    const bool   pole = (g.cflag[c] & kPole) != 0;
    const int    n    = (g.cflag[c] & kRing5) ? 5 : 6;
    for (int o = 0; o < 2; o++) {
        double w[12];
        t.triangle(c, o, n, pole, w);
        for (int k = 0; k < 12; k++)
            tw[(size_t)(o * 12 + k) * Np + c] = pole ? 0.0 : w[k];
    }
    for (int j = 0; j < 6; j++)
        for (int k = 0; k < 3; k++)
            gw[(size_t)(j * 3 + k) * Np + c] =
                j < n ? 0.5 * (t.OA(j, k, c) + t.OA((j + n - 1) % n, k, c)) : 0.0;
}

// Edge triangle e of a tile, seen from view column / triangle ev[e] = column * 8 + j.
__global__ void edge_weights_kernel(Geometry g, const int* ev, const int* ne, int tiles, double* ew) {
    const int e = threadIdx.x, tile = blockIdx.x;
    if (e >= ne[tile])
        return;
    const int    v = ev[tile * kTriMax + e], c = v >> 3, j = v & 7;
    const TriGeo t{g.areas, g.areasTr, g.nvecti, g.nvecte, g.nvecoa, g.Np};
    double       w[12];
    t.triangle(c, j, (g.cflag[c] & kRing5) ? 5 : 6, (g.cflag[c] & kPole) != 0, w);
    for (int k = 0; k < 12; k++)
        ew[((size_t)tile * 12 + k) * kTriMax + e] = w[k];
}

// ---- copies --------------------------------------------------------------------------------------
__device__ __forceinline__ void cp_halo(double* dst, const double* src) { cp_async8(dst, src); }
__device__ __forceinline__ void cp_halo(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}
// A thread's share of a plane's copies: two neighbouring own columns (threads in groups of 128, a group
// per plane in turn) or one halo column; the source moves up a level with each copy.
template<class T> struct PlaneJob {
    const T* src;
    __device__ __forceinline__ void own(T* dst, int Np) {
        if constexpr (sizeof(T) == 8)
            cp_async16(dst, src);
        else
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                             (unsigned)__cvta_generic_to_shared(dst)),
                         "l"(src)
                         : "memory");
        src += Np;
    }
    __device__ __forceinline__ void halo(T* dst, int Np) {
        cp_halo(dst, src);
        src += Np;
    }
};

// ---- the kernels ---------------------------------------------------------------------------------
// Both roles' level ring: level i's copies are complete at iteration i, when the triangle role works on
// level i and the gradient role on level i - 1; then the barrier. Each role runs its own copy of the
// loop (so that a thread's registers hold one role's weights only), with the same sequence of barriers.
// The triangle role also issues the copies (its threads have the registers for the source pointers).
__device__ __forceinline__ void role_barrier() {
    asm volatile("bar.sync 1, %0;" ::"n"(kDivThreads) : "memory");
}
template<int kStages, int kSlotBytes, bool kTri, class Start, class Issue, class Seg, class Below,
         class Comp>
__device__ __forceinline__ void role_loop(const Geometry& g, char* ring, Start start, Issue issue,
                                          Seg seg, Below below, Comp comp) {
    const int       t0 = g.tile0 * kTileCols / kPlaneCols;
    const int       t1 = (g.col_end + kPlaneCols - 1) / kPlaneCols;
    const int       nv = g.nv;
    const long long total = (long long)(t1 - t0) * nv;
    int             u     = (int)(total * blockIdx.x / gridDim.x);
    const int       u1    = (int)(total * (blockIdx.x + 1) / gridDim.x);
    bool            first = true;
    step_begin();
    while (u < u1) {
        const int       tile = t0 + u / nv, l0 = u % nv, n = min(nv - l0, u1 - u);
        const PlaneTile t    = plane_tile<PITCH, kTri ? kPlaneCols : 0>(g, tile);
        seg(t, tile);
        if (first) // the tables and weights above are nobody's to write
            step_wait();
        first = false;
        if constexpr (kTri) {
            start(t, l0);
#pragma unroll
            for (int k = 0; k < kStages - 2; k++) {
                if (k < n)
                    issue(ring + k * kSlotBytes);
                cp_async_commit();
            }
        }
        below(t, tile, l0);
        int cur = 0, prev = kStages - 1, next = kStages - 2;
        for (int i = 0; i <= n; i++) {
            if constexpr (kTri)
                cp_async_wait<kStages - 3>();
            role_barrier(); // level i is copied, D of level i - 1 written, slot `next` read
            if constexpr (kTri) {
                if (i + kStages - 2 < n)
                    issue(ring + next * kSlotBytes);
                cp_async_commit();
                if (i < n)
                    comp(t, ring + cur * kSlotBytes, l0 + i, i & 1);
            }
            else
                comp(t, ring + cur * kSlotBytes, ring + prev * kSlotBytes, l0 + i, i, i < n, i > 0);
            prev = cur;
            cur  = cur + 1 == kStages ? 0 : cur + 1;
            next = next + 1 == kStages ? 0 : next + 1;
        }
        if constexpr (kTri)
            cp_async_wait<0>();
        role_barrier();
        u += n;
    }
}

// sum over a triangle's vertices of weight . vector, from the three vectors
template<class F>
__device__ __forceinline__ double tri_dot(F weight, const double* v0, const double* v1, const double* v2) {
    double r = 0.0;
#pragma unroll
    for (int k = 0; k < 3; k++)
        r = fma(weight(k), v0[k], r);
#pragma unroll
    for (int k = 0; k < 3; k++)
        r = fma(weight(3 + k), v1[k], r);
#pragma unroll
    for (int k = 0; k < 3; k++)
        r = fma(weight(6 + k), v2[k], r);
    return r;
}
// A triangle thread (threads 256..511, x = thread - 256): the weights of its column's two triangles and
// the slots of their vertices (the column, ring points 1, 2, 3).
template<bool kW> struct TriRole {
    double w[2][9], a[kW ? 2 : 1][3];
    int    s[4];
    int    out; // slot of the first triangle's divergence (the second's kTriPlane on)
    __device__ __forceinline__ void load(const Geometry& g, const PlaneTile& t) {
        const int x  = (int)threadIdx.x - kPlaneCols;
        const int cc = min(t.c0 + x, g.N - 1);
#pragma unroll
        for (int o = 0; o < 2; o++) {
#pragma unroll
            for (int k = 0; k < 9; k++)
                w[o][k] = __ldg(g.triw + (size_t)(o * 12 + k) * g.Np + cc);
            if constexpr (kW)
#pragma unroll
                for (int k = 0; k < 3; k++)
                    a[o][k] = __ldg(g.triw + (size_t)(o * 12 + 9 + k) * g.Np + cc);
        }
        s[0] = own_slot<PITCH>(x);
        out  = tri_slot(0, x & 15, x >> 4);
#pragma unroll
        for (int j = 0; j < 3; j++)
            s[1 + j] = (int)((g.pnb[(j >> 1) * g.Np + cc] >> (16 * (j & 1))) & 0xffffu);
    }
};
// The thread of edge triangle e: its vertices' slots; the weights in shared memory (w [12][kTriMax],
// written and read by the thread itself).
template<bool kW> struct EdgeRole {
    int  s[3], out;
    bool on;
    const double* w;
    __device__ __forceinline__ void load(const Geometry& g, int tile, double* ew, int e) {
        on = e >= 0 && e < g.ptri_n[tile];
        if (!on)
            return;
        const unsigned long long v = g.ptri_v[tile * kTriMax + e];
#pragma unroll
        for (int j = 0; j < 3; j++)
            s[j] = (int)((v >> (16 * j)) & 0xffffu);
        out = (int)(v >> 48);
        for (int k = 0; k < (kW ? 12 : 9); k++)
            ew[k * kTriMax + e] = __ldg(g.ptri_w + ((size_t)tile * 12 + k) * kTriMax + e);
        w = ew + e;
    }
    __device__ __forceinline__ double weight(int k) const { return w[k * kTriMax]; }
};
// A gradient thread's weights and triangle slots.
struct GradRole {
    double   w[6][3];
    unsigned s[3];
    __device__ __forceinline__ int slot(int j) const {
        return (int)((s[j >> 1] >> (16 * (j & 1))) & 0xffffu);
    }
    __device__ __forceinline__ void load(const Geometry& g, const PlaneTile& t) {
        const int cc = min(t.c, g.N - 1);
#pragma unroll
        for (int j = 0; j < 6; j++)
#pragma unroll
            for (int k = 0; k < 3; k++)
                w[j][k] = __ldg(g.gradw + (size_t)(j * 3 + k) * g.Np + cc);
#pragma unroll
        for (int k = 0; k < 3; k++)
            s[k] = g.ptri_s[k * g.Np + cc];
    }
    __device__ __forceinline__ void apply(const double* d, double* out) const {
        out[0] = out[1] = out[2] = 0.0;
#pragma unroll
        for (int j = 0; j < 6; j++) {
            const double v = d[slot(j)];
#pragma unroll
            for (int k = 0; k < 3; k++)
                out[k] = fma(w[j][k], v, out[k]);
        }
    }
};

// Pass 0: divg = grad div (M, Wh).
constexpr int kDiv0Stages = 6;
template<class TD>
__global__ void __launch_bounds__(kDivThreads, 1)
    divm0_plane_kernel(Geometry g, Phys P, const double* __restrict__ Mh,
                       const double* __restrict__ Wh, TD* __restrict__ divg) {
    extern __shared__ __align__(16) char ring[];
    constexpr int kSlotBytes = 4 * PITCH * (int)sizeof(double);
    constexpr int kStages    = kDiv0Stages;
    double*       D  = reinterpret_cast<double*>(ring + kStages * kSlotBytes); // [2][kTriPitch]
    const int     Np = g.Np, nv = g.nv, nvi = g.nvi;
    const size_t  plane = (size_t)nv * Np;
    double*       ew = D + 2 * kTriPitch;  // [12][kTriMax]
    double2*      lv = reinterpret_cast<double2*>(ew + 12 * kTriMax); // rscale, -1/dz by level
    for (int l = threadIdx.x; l < nv; l += kDivThreads)
        lv[l] = make_double2(g.lt[kLtRscale * nvi + l], -g.lt[kLtRDz * nvi + l]);
    if (threadIdx.x >= kPlaneCols) {
        TriRole<true>    r{};
        PlaneJob<double> own[2], halo[2]; // planes grp, grp + 2 of Mh x, y, z, Wh above
        const int        grp = ((int)threadIdx.x >> 7) & 1, y = ((int)threadIdx.x & 127) * 2;
        const int        ys = own_slot<PITCH>(y);
        int              hs = -1;
        bool             mine = false;
        auto start = [&](const PlaneTile& t, int l0) {
            mine = y < t.ncopy;
            const int e = (int)threadIdx.x & 127;
            hs = e < t.nh ? g.phslot[(t.c0 / kPlaneCols) * g.phmax + e] : -1;
            const int id = e < t.nh ? g.phalo[(t.c0 / kPlaneCols) * g.phmax + e] : 0;
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int     p   = grp + 2 * k;
                const double* src = (p < 3 ? Mh + p * plane : Wh + Np) + (size_t)l0 * Np;
                own[k].src  = src + t.c0 + y;
                halo[k].src = src + id;
            }
        };
        auto issue = [&](char* slot) {
            double* d = reinterpret_cast<double*>(slot) + grp * PITCH;
            if (mine)
#pragma unroll
                for (int k = 0; k < 2; k++)
                    own[k].own(d + 2 * k * PITCH + ys, Np);
            if (hs >= 0)
#pragma unroll
                for (int k = 0; k < 2; k++)
                    halo[k].halo(d + 2 * k * PITCH + hs, Np);
        };
        double wl[4] = {0, 0, 0, 0}; // Wh at the level's lower interface
        auto   seg   = [&](const PlaneTile& t, int) { r.load(g, t); };
        auto   below = [&](const PlaneTile& t, int, int l0) {
            const int c = min(t.c0 + (int)threadIdx.x - kPlaneCols, g.N - 1);
#pragma unroll
            for (int v = 0; v < 4; v++) {
                const int id = v == 0 ? c : g.nb[(size_t)(v - 1) * Np + c];
                wl[v]        = id >= 0 ? Wh[(size_t)l0 * Np + id] : 0.0;
            }
        };
        auto comp = [&](const PlaneTile&, const char* slot, int lev, int buf) {
            const double* q      = reinterpret_cast<const double*>(slot);
            const double  rscale = lv[lev].x, mdz = lv[lev].y;
            double        m[4][3], dw[4];
#pragma unroll
            for (int v = 0; v < 4; v++) {
#pragma unroll
                for (int k = 0; k < 3; k++)
                    m[v][k] = q[k * PITCH + r.s[v]];
                const double wt = q[3 * PITCH + r.s[v]];
                dw[v]           = wl[v] - wt;
                wl[v]           = wt;
            }
            double* out = D + buf * kTriPitch + r.out;
#pragma unroll
            for (int o = 0; o < 2; o++) {
                const double h = tri_dot([&](int k) { return r.w[o][k]; }, m[0], m[1 + o], m[2 + o]);
                const double w = fma(r.a[o][2], dw[2 + o], fma(r.a[o][1], dw[1 + o], r.a[o][0] * dw[0]));
                out[o * kTriPlane] = fma(rscale, h, mdz * w);
            }
        };
        role_loop<kStages, kSlotBytes, true>(g, ring, start, issue, seg, below, comp);
    }
    else {
        GradRole       r{};
        EdgeRole<true> ed{};
        double         we[3] = {0, 0, 0}; // Wh at the edge triangle's vertices, the level's lower interface
        auto           seg   = [&](const PlaneTile& t, int tile) {
            r.load(g, t);
            ed.load(g, tile, ew, threadIdx.x < kTriMax ? (int)threadIdx.x : -1);
        };
        auto below = [&](const PlaneTile&, int tile, int l0) {
            if (ed.on) {
                const int view = g.ptri_view[tile * kTriMax + threadIdx.x], c = view >> 3, j = view & 7;
                const int n = (g.cflag[c] & kRing5) ? 5 : 6;
                we[0] = Wh[(size_t)l0 * Np + c];
                we[1] = Wh[(size_t)l0 * Np + g.ring[(size_t)j * Np + c]];
                we[2] = Wh[(size_t)l0 * Np + g.ring[(size_t)((j + 1) % n) * Np + c]];
            }
        };
        auto comp = [&](const PlaneTile& t, const char* slot, const char*, int lev, int i, bool tri,
                        bool grad) {
            if (tri && ed.on) { // the edge triangles of this level, beside the triangle role
                const double* q = reinterpret_cast<const double*>(slot);
                double        m[3][3], dw[3];
#pragma unroll
                for (int v = 0; v < 3; v++) {
#pragma unroll
                    for (int k = 0; k < 3; k++)
                        m[v][k] = q[k * PITCH + ed.s[v]];
                    const double wt = q[3 * PITCH + ed.s[v]];
                    dw[v]           = we[v] - wt;
                    we[v]           = wt;
                }
                const double h = tri_dot([&](int k) { return ed.weight(k); }, m[0], m[1], m[2]);
                const double w = fma(ed.weight(11), dw[2], fma(ed.weight(10), dw[1], ed.weight(9) * dw[0]));
                D[(i & 1) * kTriPitch + ed.out] = fma(lv[lev].x, h, lv[lev].y * w);
            }
            if (grad) { // the gradient of the level below
                const double rscale = lv[lev - 1].x;
                double       o[3];
                r.apply(D + ((i - 1) & 1) * kTriPitch, o);
                if (t.store)
#pragma unroll
                    for (int k = 0; k < 3; k++)
                        divg[k * plane + (size_t)(lev - 1) * Np + t.c] = (TD)(rscale * o[k]);
            }
        };
        role_loop<kStages, kSlotBytes, false>(g, ring, 0, 0, seg, below, comp);
    }
}

// Horizontal momentum of a small step (kSlow false): pass 1 of the damping on divg, the pressure gradient
// of the deviations, the slow tendency; the radial component removed from their sum. Or the slow
// tendency itself (kSlow, once per RK stage; the momentum part of Compute_Slow_Modes / _Poles,
// src/headers/dyn/thor_slowmodes.h:48-683): the same with the stage's pressure, minus the advection,
// plus the diffusion; it also leaves what the rest of the slow modes needs of the gradient and the
// advection: fx the work of the pressure gradient, fy the radial advection. kSlow: 95 us at glevel 6, 48
// levels; the column-tile kernel, with the flux divergences and the vertical parts that stage_kernel now
// completes, 280.
constexpr int kMomStages = 6, kSlowStages = 5;
template<class TD, bool kSlow>
__global__ void __launch_bounds__(kDivThreads, 1)
    momentum_plane_kernel(Geometry g, Phys P, State s, double dt, bool damp) {
    extern __shared__ __align__(16) char ring[];
    // a slot: ps (gathered), the own planes SlowMh, Mhs (kSlow: pk; Adv, diffmh, Mhk, Rhok), then divg
    // (gathered)
    constexpr int kOwn = kSlow ? 10 : 6, kHalf = kOwn / 2;
    constexpr int kDouble    = PITCH + kOwn * kPlaneCols;
    constexpr int kSlotBytes = kDouble * (int)sizeof(double) + 3 * PITCH * (int)sizeof(TD);
    constexpr int kStages    = kSlow ? kSlowStages : kMomStages;
    static_assert(kSlotBytes % 16 == 0, "slots keep 16-byte alignment");
    double*      D  = reinterpret_cast<double*>(ring + kStages * kSlotBytes);
    const int    Np = g.Np, nv = g.nv, nvi = g.nvi;
    const size_t plane = (size_t)nv * Np;
    const TD*    divg  = reinterpret_cast<const TD*>(s.divg);
    const double* press = kSlow ? s.pk : s.ps;
    double*      ew    = D + 2 * kTriPitch; // [9][kTriMax]
    double2*     lv    = reinterpret_cast<double2*>(ew + 9 * kTriMax); // rscale, Kdhz by level
    for (int l = threadIdx.x; l < nv; l += kDivThreads)
        lv[l] = make_double2(g.lt[kLtRscale * nvi + l], g.Kdhz[l]);
    if (threadIdx.x >= kPlaneCols) {
        TriRole<false>   r{};
        PlaneJob<double> ps, po[kHalf], hp;    // ps (group 0), half of the own planes
        PlaneJob<TD>     pd[2], hd[2];         // divg grp (and 2: group 0)
        const int        x = (int)threadIdx.x - kPlaneCols, grp = x >> 7, y = (x & 127) * 2;
        const int        ys = own_slot<PITCH>(y);
        int              hs = -1;
        bool             mine = false;
        // group 0: ps, divg z and the first half of the own planes; group 1: divg x, y and the others
        auto start = [&](const PlaneTile& t, int l0) {
            const size_t off = (size_t)l0 * Np;
            mine             = y < t.ncopy;
            const int e      = x & 127;
            hs               = e < t.nh ? g.phslot[(t.c0 / kPlaneCols) * g.phmax + e] : -1;
            const int id     = e < t.nh ? g.phalo[(t.c0 / kPlaneCols) * g.phmax + e] : 0;
            ps.src           = press + off + t.c0 + y;
            hp.src           = press + off + id;
#pragma unroll
            for (int k = 0; k < kHalf; k++) {
                const double* src;
                if (kSlow) { // Adv, diffmh x, y | diffmh z, Mhk, Rhok
                    if (grp == 0)
                        src = k < 3 ? s.Adv + k * plane : s.diffmh + (k - 3) * plane;
                    else
                        src = k == 0 ? s.diffmh + 2 * plane : k < 4 ? s.Mhk + (k - 1) * plane : s.Rhok;
                }
                else
                    src = (grp ? s.Mhs : s.SlowMh) + k * plane;
                po[k].src = src + off + t.c0 + y;
            }
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const TD* d = divg + (grp ? k : 2) * plane + off;
                pd[k].src   = d + t.c0 + y;
                hd[k].src   = d + id;
            }
        };
        auto issue = [&](char* slot) {
            double* d  = reinterpret_cast<double*>(slot);
            TD*     dg = reinterpret_cast<TD*>(d + kDouble);
            if (mine) {
#pragma unroll
                for (int k = 0; k < kHalf; k++)
                    po[k].own(d + PITCH + (kHalf * grp + k) * kPlaneCols + y, Np);
                if (grp == 0) {
                    ps.own(d + ys, Np);
                    if (damp)
                        pd[0].own(dg + 2 * PITCH + ys, Np);
                }
                else if (damp) {
                    pd[0].own(dg + ys, Np);
                    pd[1].own(dg + PITCH + ys, Np);
                }
            }
            if (hs >= 0) {
                if (grp == 0) {
                    hp.halo(d + hs, Np);
                    if (damp)
                        hd[0].halo(dg + 2 * PITCH + hs, Np);
                }
                else if (damp) {
                    hd[0].halo(dg + hs, Np);
                    hd[1].halo(dg + PITCH + hs, Np);
                }
            }
        };
        // the edge triangles on the two warps without halo columns to copy
        EdgeRole<false> ed{};
        const int       e    = ((x >> 5) & 3) == 3 ? (x & 31) + 32 * grp : -1;
        auto            seg  = [&](const PlaneTile& t, int tile) {
            r.load(g, t);
            ed.load(g, tile, ew, e);
        };
        auto below = [](const PlaneTile&, int, int) {};
        auto comp = [&](const PlaneTile&, const char* slot, int lev, int buf) {
            if (!damp)
                return;
            const TD* q = reinterpret_cast<const TD*>(reinterpret_cast<const double*>(slot) + kDouble);
            const double rscale = lv[lev].x;
            double       m[4][3];
            auto         vertex = [&](int sl, double* mv) {
#pragma unroll
                for (int k = 0; k < 3; k++)
                    mv[k] = (double)q[k * PITCH + sl];
            };
#pragma unroll
            for (int v = 0; v < 4; v++)
                vertex(r.s[v], m[v]);
            double* out = D + buf * kTriPitch;
#pragma unroll
            for (int o = 0; o < 2; o++)
                out[r.out + o * kTriPlane] =
                    rscale * tri_dot([&](int k) { return r.w[o][k]; }, m[0], m[1 + o], m[2 + o]);
            if (ed.on) {
#pragma unroll
                for (int v = 0; v < 3; v++)
                    vertex(ed.s[v], m[v]);
                out[ed.out] = rscale * tri_dot([&](int k) { return ed.weight(k); }, m[0], m[1], m[2]);
            }
        };
        role_loop<kStages, kSlotBytes, true>(g, ring, start, issue, seg, below, comp);
    }
    else {
        GradRole r{};
        double   gd[7][3] = {}, fr[3] = {};
        auto     below = [](const PlaneTile&, int, int) {};
        auto     seg = [&](const PlaneTile& t, int) {
            r.load(g, t);
            const bool valid = t.c < g.N;
#pragma unroll
            for (int j = 0; j < 7; j++) {
                const bool use = valid && (j == 0 || t.point(j) != t.own); // not a hole
#pragma unroll
                for (int k = 0; k < 3; k++)
                    gd[j][k] = use ? __ldg(g.grad + (size_t)(j * 3 + k) * Np + t.c) : 0.0;
            }
#pragma unroll
            for (int k = 0; k < 3; k++)
                fr[k] = valid ? __ldg(g.func_r + (size_t)k * Np + t.c) : 0.0;
        };
        auto one = [&](const PlaneTile& t, const char* slot, int lev, const double* d, bool store) {
            const double* q      = reinterpret_cast<const double*>(slot);
            const double  rscale = lv[lev].x;
            double        a[3]   = {0, 0, 0}, l[3] = {0, 0, 0};
#pragma unroll
            for (int j = 0; j < 7; j++) {
                const double pv = q[t.point(j)];
#pragma unroll
                for (int k = 0; k < 3; k++)
                    a[k] = fma(gd[j][k], pv, a[k]);
            }
            if (damp)
                r.apply(d, l);
            const double* o  = q + PITCH + threadIdx.x;
            const double  kd = lv[lev].y;
            double        T[3];
            if constexpr (kSlow) {
                const size_t i   = (size_t)lev * Np + t.c;
                const double rho = o[9 * kPlaneCols];
                double       adv[3], M[3], gp = 0.0, gm = 0.0, mr = 0.0;
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    adv[k] = o[k * kPlaneCols];
                    M[k]   = o[(6 + k) * kPlaneCols];
                    T[k]   = fma(-rscale, fma(kd, l[k], a[k]), -adv[k]);
                    gp     = fma(a[k], fr[k], gp);
                    gm     = fma(a[k], M[k], gm);
                    mr     = fma(M[k], fr[k], mr);
                }
                const double vr = T[0] * fr[0] + T[1] * fr[1] + T[2] * fr[2];
                if (!store)
                    return;
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    double v = fma(-vr, fr[k], T[k]) + o[(3 + k) * kPlaneCols];
                    if (P.drag) // modules' and the explicit sponge's tendency
                        v += s.dMh[k * plane + i];
                    s.SlowMh[k * plane + i] = v;
                }
                s.fx[i] = rscale * fma(-gp, mr, gm) / rho; // the tangential gradient times M / rho
                if (P.NonHydro)
                    s.fy[i] = adv[0] * fr[0] + adv[1] * fr[1] + adv[2] * fr[2];
                else
                    s.fy[i] = (M[0] * M[0] + M[1] * M[1] + M[2] * M[2]) / (rho * (g.Altitude[lev] + P.A));
                return;
            }
#pragma unroll
            for (int k = 0; k < 3; k++)
                T[k] = fma(-rscale, fma(kd, l[k], a[k]), o[k * kPlaneCols]) * dt;
            const double vr = T[0] * fr[0] + T[1] * fr[1] + T[2] * fr[2];
            if (store)
#pragma unroll
                for (int k = 0; k < 3; k++)
                    s.Mhs[k * plane + (size_t)lev * Np + t.c] =
                        o[(3 + k) * kPlaneCols] + fma(-vr, fr[k], T[k]);
        };
        auto comp = [&](const PlaneTile& t, const char*, const char* below, int lev, int i, bool,
                        bool grad) {
            if (grad)
                one(t, below, lev - 1, D + ((i - 1) & 1) * kTriPitch, t.store);
        };
        role_loop<kStages, kSlotBytes, false>(g, ring, 0, 0, seg, below, comp);
    }
}

template<class TD>
void launch_divm0_t(const Geometry& g, const Phys& P, const double* M, const double* W, double* divg,
                    cudaStream_t st) {
    const size_t smem =
        sizeof(double) * (kDiv0Stages * 4 * PITCH + 2 * kTriPitch + 12 * kTriMax + 2 * g.nv);
    static SmemOptIn opt;
    if (opt.ensure(divm0_plane_kernel<TD>, smem) == cudaSuccess)
        launch_step(divm0_plane_kernel<TD>, plane_ctas(g, 1), kDivThreads, smem, st, g, P, M, W,
                    reinterpret_cast<TD*>(divg));
}
template<class TD, bool kSlow>
void launch_momentum_t(const Geometry& g, const Phys& P, const State& s, double dt, bool damp,
                       cudaStream_t st) {
    const size_t smem = (kSlow ? kSlowStages : kMomStages)
                            * (sizeof(double) * (PITCH + (kSlow ? 10 : 6) * kPlaneCols) + sizeof(TD) * 3 * PITCH)
                        + sizeof(double) * (2 * kTriPitch + 9 * kTriMax + 2 * g.nv);
    static SmemOptIn opt;
    if (opt.ensure(momentum_plane_kernel<TD, kSlow>, smem) == cudaSuccess)
        launch_step(momentum_plane_kernel<TD, kSlow>, plane_ctas(g, 1), kDivThreads, smem, st, g, P, s, dt,
                    damp && P.DivDampP);
}

// ---------------------------------------------------------------------------------------------
// Advection and Coriolis of an RK stage (Compute_Advec_Cori1 / _Poles, Compute_Advec_Cori2,
// src/headers/dyn/thor_adv_cor.h:51-536). The cartesian velocity v = M / rho + (w / rho) r^ of a column
// is formed once per level in shared memory (own columns and halo), where the column-tile form formed
// it at each of the seven points; the flux divergence is sum_j v_j (div_j . M_j). The velocities run
// one level ahead, so that the vertical flux has the level above at hand. glevel 6, 48 levels: 140 us with
// thermo_kernel (the column-tile kernel of both 272); bound by the shared-memory reads, 42 a cell, and the
// five gathered planes' halo copies (these over all warps: 145 -> 154 us).
// ---------------------------------------------------------------------------------------------
constexpr int kAdvStages = 4, kAdvSlot = 5 * PITCH + kPlaneCols;
__global__ void __launch_bounds__(kPlaneCols, 2) adv_plane_kernel(Geometry g, Phys P, State s) {
    extern __shared__ __align__(16) double ringd[];
    double*      sv = ringd + kAdvStages * kAdvSlot; // [2][3][PITCH]
    const int    Np = g.Np, nv = g.nv, nvi = g.nvi, x = threadIdx.x;
    const size_t plane = (size_t)nv * Np;
    const double* lt   = g.lt;
    const double  Omega = P.Omega;
    double        d[7][3], fr[3], frh[3], vprev[3], vcur[3], vnext[3], whl = 0.0;
    const double* const src[6] = {s.Mhk, s.Mhk + plane, s.Mhk + 2 * plane, s.Rhok, s.Wk, s.Whk + Np};
    auto vel = [&](double m0, double m1, double m2, double rho, double w, const double* f, double* v) {
        const double yr = 1.0 / rho, wr = div_rcp(w, rho, yr);
        v[0] = fma(wr, f[0], div_rcp(m0, rho, yr));
        v[1] = fma(wr, f[1], div_rcp(m1, rho, yr));
        v[2] = fma(wr, f[2], div_rcp(m2, rho, yr));
    };
    auto seg = [&](const PlaneTile& t) {
        const bool valid = t.c < g.N;
        const int  c     = min(t.c, g.N - 1);
#pragma unroll
        for (int j = 0; j < 7; j++) {
            const bool use = valid && (j == 0 || t.point(j) != t.own); // not a hole
#pragma unroll
            for (int k = 0; k < 3; k++)
                d[j][k] = use ? __ldg(g.div + (size_t)(j * 3 + k) * Np + c) : 0.0;
        }
#pragma unroll
        for (int k = 0; k < 3; k++) {
            fr[k]  = __ldg(g.func_r + (size_t)k * Np + c);
            frh[k] = t.hid >= 0 ? __ldg(g.func_r + (size_t)k * Np + t.hid) : 0.0;
            vnext[k] = 0.0;
            vcur[k]  = 0.0;
        }
    };
    auto below = [&](const PlaneTile& t, int l0) {
        const int c = min(t.c, g.N - 1);
        if (l0 > 0) { // the velocity below the range
            const size_t i = (size_t)(l0 - 1) * Np + c;
            vel(s.Mhk[i], s.Mhk[plane + i], s.Mhk[2 * plane + i], s.Rhok[i], s.Wk[i], fr, vnext);
        }
        whl = s.Whk[(size_t)l0 * Np + c];
    };
    auto prep = [&](const PlaneTile& t, double* b, int, int buf) {
        double* v = sv + buf * 3 * PITCH;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            vprev[k] = vcur[k];
            vcur[k]  = vnext[k];
        }
        const double* q = b + t.own;
        vel(q[0], q[PITCH], q[2 * PITCH], q[3 * PITCH], q[4 * PITCH], fr, vnext);
#pragma unroll
        for (int k = 0; k < 3; k++)
            v[k * PITCH + t.own] = vnext[k];
        if (t.hid >= 0) {
            const double* h = b + t.hslot;
            double        vh[3];
            vel(h[0], h[PITCH], h[2 * PITCH], h[3 * PITCH], h[4 * PITCH], frh, vh);
#pragma unroll
            for (int k = 0; k < 3; k++)
                v[k * PITCH + t.hslot] = vh[k];
        }
    };
    auto comp = [&](const PlaneTile& t, const double* b, int lev, int buf) {
        // prep has moved on: vcur is this level's velocity if a level above was prepared
        const bool    above = lev < nv - 1;
        const double* v     = sv + buf * 3 * PITCH;
        double        sum[3] = {0, 0, 0}, v0[3];
#pragma unroll
        for (int j = 0; j < 7; j++) {
            const double* q = b + t.point(j);
            const double* w = v + t.point(j);
            const double  f = fma(d[j][2], q[2 * PITCH], fma(d[j][1], q[PITCH], d[j][0] * q[0]));
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const double vj = w[k * PITCH];
                sum[k]          = fma(f, vj, sum[k]);
                if (j == 0)
                    v0[k] = vj;
            }
        }
        const double wht = b[5 * PITCH + x];
        if (t.store) {
            const double rscale = lt[kLtRscale * nvi + lev], rho = b[3 * PITCH + t.own];
            double       r2p = 1.0, r2l = 1.0, C[3];
            if (P.DeepModel) {
                r2p  = lt[kLtR2hD * nvi + lev + 1];
                r2l  = lt[kLtR2hD * nvi + lev];
                C[0] = -2.0 * Omega * v0[1] * rho;
                C[1] = 2.0 * Omega * v0[0] * rho;
                C[2] = 0.0;
            }
            else {
                C[0] = 2 * Omega * (v0[2] * fr[2] * fr[1] - v0[1] * (fr[2] * fr[2])) * rho;
                C[1] = -2 * Omega * (v0[2] * fr[2] * fr[0] - v0[0] * (fr[2] * fr[2])) * rho;
                C[2] = 2 * Omega * (v0[1] * fr[2] * fr[0] - v0[0] * fr[2] * fr[1]) * rho;
            }
            const double dz = -lt[(P.DeepModel ? kLtRDzR2m : kLtRDz) * nvi + lev];
#pragma unroll
            for (int k = 0; k < 3; k++) {
                double lo = 0.0, hi = 0.0;
                if (lev > 0)
                    lo = ((above ? vprev[k] : vcur[k]) * lt[kLtHIntt * nvi + lev]
                          + v0[k] * lt[kLtHIntl * nvi + lev]) * whl;
                if (above)
                    hi = (v0[k] * lt[kLtHIntt * nvi + lev + 1] + vnext[k] * lt[kLtHIntl * nvi + lev + 1])
                         * wht;
                s.Adv[k * plane + (size_t)lev * Np + t.c] =
                    fma(rscale, sum[k], fma(lo * r2l - hi * r2p, dz, C[k]));
            }
        }
        whl = wht;
    };
    lag_loop<5, 1, kAdvStages, true>(g, ringd, src, seg, below, prep, comp);
}

// ---------------------------------------------------------------------------------------------
// A hyperdiffusion pass (Diffusion_Op + Diffusion_Op_Poles, src/headers/dyn/thor_diff.h:54-880, and
// Correct_Horizontal, :882-915, on the last): the Laplacian's 7 weights per column stay in registers
// and serve the six variables. kFirst: the arguments rho, v, w, Rd T (or Cv T) are formed once per
// column in the ring (own columns and halo), where each of the seven points formed them before. The
// pass before the last stores its result times rho for v, w and T, which is the last one's argument.
// glevel 6, 48 levels, first and last pass: 64 and 61 us (the column-tile form 161 and 118), bound by the
// 6 gathered planes' copies: 12 and 13 planes of bytes alone are 28 and 31 us.
// ---------------------------------------------------------------------------------------------
constexpr int kDiffStages = 4, kDiffSlot = 6 * PITCH;
template<bool kFirst, bool kUni>
__global__ void __launch_bounds__(kPlaneCols, 2)
    diffusion_plane_kernel(Geometry g, Phys P, State s, const double* __restrict__ in,
                           double* __restrict__ out, bool last, bool scale) {
    extern __shared__ __align__(16) double ringd[];
    const int    Np = g.Np, nv = g.nv, nvi = g.nvi, x = threadIdx.x;
    const size_t plane = (size_t)nv * Np;
    double       w[7];
    int          pt[6];
    const double* const src[6] = {kFirst ? s.Rhok : in,
                                  kFirst ? s.Mhk : in + plane,
                                  kFirst ? s.Mhk + plane : in + 2 * plane,
                                  kFirst ? s.Mhk + 2 * plane : in + 3 * plane,
                                  kFirst ? s.Wk : in + 4 * plane,
                                  kFirst ? s.T : in + 5 * plane};
    auto below = [](const PlaneTile&, int) {};
    auto seg = [&](const PlaneTile& t) {
        const int c = min(t.c, g.N - 1);
        // the ring: the stencil points, without a pentagon's repeated one
        const bool five = (g.cflag[c] & kRing5) != 0;
#pragma unroll
        for (int j = 0; j < 7; j++)
            w[j] = j == 6 && five ? 0.0 : __ldg(g.lapw + (size_t)j * Np + c);
#pragma unroll
        for (int j = 0; j < 6; j++)
            pt[j] = t.point(j + 1);
    };
    auto prep = [&](const PlaneTile& t, double* b, int lev, int) {
        auto convert = [&](double* q, int id) {
            const double rho = q[0], yr = 1.0 / rho;
#pragma unroll
            for (int k = 1; k < 5; k++)
                q[k * PITCH] = div_rcp(q[k * PITCH], rho, yr);
            const int    i  = lev * Np + id;
            const double Rd = rd_at<kUni>(P, s, i);
            q[5 * PITCH] *= P.energy ? cp_at<kUni>(P, s, i) - Rd : Rd;
        };
        if constexpr (kFirst) {
            if (x < t.ncopy)
                convert(b + t.own, t.c);
            if (t.hid >= 0)
                convert(b + t.hslot, t.hid);
        }
    };
    auto comp = [&](const PlaneTile& t, const double* b, int lev, int) {
        double a0[6], acc[6];
#pragma unroll
        for (int v = 0; v < 6; v++) {
            a0[v]  = b[v * PITCH + t.own];
            acc[v] = w[0] * a0[v];
        }
#pragma unroll
        for (int j = 0; j < 6; j++)
#pragma unroll
            for (int v = 0; v < 6; v++)
                acc[v] = fma(w[j + 1], b[v * PITCH + pt[j]] - a0[v], acc[v]);
        if (!t.store)
            return;
        const double rscale = g.lt[kLtRscale * nvi + lev], sc = rscale * rscale;
        const size_t i = (size_t)lev * Np + t.c;
        if (!last) {
            const double r = scale ? (kFirst ? a0[0] : s.Rhok[i]) : 1.0;
            out[i]         = acc[0] * sc;
#pragma unroll
            for (int v = 1; v < 6; v++)
                out[v * plane + i] = acc[v] * sc * r;
            return;
        }
        const double sd = ((P.HyDiffOrder / 2) & 1 ? 1.0 : -1.0) * g.Kdh4[lev] * sc; // -(-1)^(order/2) Kdh4
#pragma unroll
        for (int v = 0; v < 6; v++)
            acc[v] *= sd;
        double fr[3];
#pragma unroll
        for (int k = 0; k < 3; k++)
            fr[k] = __ldg(g.func_r + (size_t)k * Np + t.c);
        // Correct_Horizontal: remove the radial component of the momentum diffusion
        const double r = fma(fr[2], acc[3], fma(fr[1], acc[2], fr[0] * acc[1]));
        s.diffrh[i]    = acc[0];
#pragma unroll
        for (int k = 0; k < 3; k++)
            s.diffmh[k * plane + i] = fma(-fr[k], r, acc[1 + k]);
        s.diffw[i]  = acc[4];
        s.diffpr[i] = acc[5];
    };
    lag_loop<6, 0, kDiffStages, false>(g, ringd, src, seg, below, prep, comp);
}

template<bool kFirst, bool kUni>
void launch_diffusion_t(const Geometry& g, const Phys& P, const State& s, const double* in, double* out,
                        bool last, bool scale, cudaStream_t st) {
    constexpr size_t smem = sizeof(double) * kDiffStages * kDiffSlot;
    static SmemOptIn opt;
    if (opt.ensure(diffusion_plane_kernel<kFirst, kUni>, smem) == cudaSuccess)
        launch_step(diffusion_plane_kernel<kFirst, kUni>, plane_ctas(g, 2), kPlaneCols, smem, st, g, P, s,
                    in, out, last, scale);
}

} // namespace

void launch_adv_planes(const Geometry& g, const Phys& P, const State& s, cudaStream_t st) {
    constexpr size_t smem = sizeof(double) * (kAdvStages * kAdvSlot + 6 * PITCH);
    static SmemOptIn opt;
    if (opt.ensure(adv_plane_kernel, smem) == cudaSuccess)
        launch_step(adv_plane_kernel, plane_ctas(g, 2), kPlaneCols, smem, st, g, P, s);
}
void launch_diffusion_planes(const Geometry& g, const Phys& P, const State& s, int stepnum, bool last,
                             bool before_last, cudaStream_t st) {
    // passes alternate between the two halves of the diff buffer
    const size_t  plane6 = (size_t)6 * g.nv * g.Np;
    const double* in     = s.diff + ((stepnum + 1) % 2) * plane6;
    double*       out    = s.diff + (stepnum % 2) * plane6;
    if (stepnum > 0)
        launch_diffusion_t<false, true>(g, P, s, in, out, last, before_last, st);
    else if (P.uniform_thermo)
        launch_diffusion_t<true, true>(g, P, s, in, out, last, before_last, st);
    else
        launch_diffusion_t<true, false>(g, P, s, in, out, last, before_last, st);
}

void launch_divm0_planes(const Geometry& g, const Phys& P, const State& s, bool small_step,
                         cudaStream_t st) {
    const double *M = small_step ? s.Mhs : s.Mhk, *W = small_step ? s.Whs : s.Whk;
    if (P.mixed && kDivgF32)
        launch_divm0_t<float>(g, P, M, W, s.divg, st);
    else
        launch_divm0_t<double>(g, P, M, W, s.divg, st);
}
void launch_momentum_planes(const Geometry& g, const Phys& P, const State& s, double dt, bool damp,
                            cudaStream_t st) {
    if (P.mixed && kDivgF32)
        launch_momentum_t<float, false>(g, P, s, dt, damp, st);
    else
        launch_momentum_t<double, false>(g, P, s, dt, damp, st);
}
void launch_slow_momentum(const Geometry& g, const Phys& P, const State& s, cudaStream_t st) {
    if (P.mixed && kDivgF32)
        launch_momentum_t<float, true>(g, P, s, 0.0, true, st);
    else
        launch_momentum_t<double, true>(g, P, s, 0.0, true, st);
}

void launch_tri_weights(const Geometry& g, int tiles, double* tw, double* gw, double* ew,
                        cudaStream_t st) {
    tri_weights_kernel<<<(g.N + 127) / 128, 128, 0, st>>>(g, tw, gw);
    edge_weights_kernel<<<tiles, kTriMax, 0, st>>>(g, g.ptri_view, g.ptri_n, tiles, ew);
}

} // namespace thorx
