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
// column; the first 64 threads also take an edge triangle, its weights in shared memory); the gradient
// runs one level behind the triangles, so a level costs one barrier. 16 warps, so that every scheduler
// has four and a thread may hold 128 registers: with warps of their own for the edge triangles a
// scheduler had five and the weights spilled.
#include "dyn_common.cuh"
#include "planes.cuh"

namespace thorx {
namespace {

constexpr int kDivThreads = 2 * kPlaneCols;
constexpr int kTriPitch   = 2 * kPlaneCols + kTriMax;            // D of a level: U, V, edge
constexpr int PITCH       = kPitchRhombus;

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
// One level plane (own columns; halo when kHalo) into dst, by the threads x0 .. x0 + 127 and, for the
// halo, the first nh threads.
template<bool kHalo, class T>
__device__ __forceinline__ void plane_copy(const Geometry& g, const PlaneTile& t, T* dst,
                                           const T* __restrict__ plane, int x0) {
    constexpr int kVec = 16 / sizeof(T);
    const int     y    = ((int)threadIdx.x - x0) * kVec;
    if (y >= 0 && y < t.ncopy)
        cp_async16(dst + y, plane + t.c0 + y);
    if (kHalo)
        if (t.hid >= 0)
            cp_halo(dst + kPlaneCols + threadIdx.x, plane + t.hid);
}

// ---- the kernels ---------------------------------------------------------------------------------
// Both roles' level ring: level i's copies are complete at iteration i, when the triangle role works on
// level i and the gradient role on level i - 1; then the barrier. Each role runs its own copy of the
// loop (so that a thread's registers hold one role's weights only), with the same sequence of barriers.
__device__ __forceinline__ void role_barrier() {
    asm volatile("bar.sync 1, %0;" ::"n"(kDivThreads) : "memory");
}
template<int kStages, int kSlotBytes, bool kTri, class Issue, class Seg, class Comp>
__device__ __forceinline__ void role_loop(const Geometry& g, char* ring, Issue issue, Seg seg,
                                          Comp comp) {
    const int       t0 = g.tile0 * kTileCols / kPlaneCols;
    const int       t1 = (g.col_end + kPlaneCols - 1) / kPlaneCols;
    const int       nv = g.nv;
    const long long total = (long long)(t1 - t0) * nv;
    int             u     = (int)(total * blockIdx.x / gridDim.x);
    const int       u1    = (int)(total * (blockIdx.x + 1) / gridDim.x);
    while (u < u1) {
        const int       tile = t0 + u / nv, l0 = u % nv, n = min(nv - l0, u1 - u);
        const PlaneTile t    = plane_tile(g, tile);
#pragma unroll
        for (int k = 0; k < kStages - 2; k++) {
            if (k < n)
                issue(t, ring + k * kSlotBytes, l0 + k);
            cp_async_commit();
        }
        seg(t, tile, l0);
        int cur = 0, prev = kStages - 1, next = kStages - 2;
        for (int i = 0; i <= n; i++) {
            cp_async_wait<kStages - 3>();
            role_barrier(); // level i is copied, D of level i - 1 written, slot `next` read
            if (i + kStages - 2 < n)
                issue(t, ring + next * kSlotBytes, l0 + i + kStages - 2);
            cp_async_commit();
            if (kTri ? i < n : i > 0) {
                if (kTri)
                    comp(t, ring + cur * kSlotBytes, l0 + i, i & 1);
                else
                    comp(t, ring + prev * kSlotBytes, l0 + i - 1, (i - 1) & 1);
            }
            prev = cur;
            cur  = cur + 1 == kStages ? 0 : cur + 1;
            next = next + 1 == kStages ? 0 : next + 1;
        }
        cp_async_wait<0>();
        role_barrier();
        u += n;
    }
}

// A triangle thread (threads 256..511, x = thread - 256): the weights of its column's two triangles,
// the slots of their vertices (the column, ring points 1, 2, 3); for x < 64 also an edge triangle's
// vertices (weights in ew [12][kTriMax], written and read by the thread itself).
template<bool kW> struct TriRole {
    double w[2][9], a[kW ? 2 : 1][3];
    int    s[4], e[3];
    bool   edge;
    __device__ __forceinline__ void load(const Geometry& g, const PlaneTile& t, int tile, double* ew) {
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
        s[0] = x;
#pragma unroll
        for (int j = 0; j < 3; j++)
            s[1 + j] = (int)((g.pnb[(j >> 1) * g.Np + cc] >> (16 * (j & 1))) & 0xffffu);
        edge = x < g.ptri_n[tile];
        if (edge) {
            const unsigned long long v = g.ptri_v[tile * kTriMax + x];
#pragma unroll
            for (int j = 0; j < 3; j++)
                e[j] = (int)((v >> (16 * j)) & 0xffffu);
            for (int k = 0; k < (kW ? 12 : 9); k++)
                ew[k * kTriMax + x] = __ldg(g.ptri_w + ((size_t)tile * 12 + k) * kTriMax + x);
        }
    }
    // sum over a triangle's vertices of weight . vector, from the three vectors
    template<class F>
    __device__ static __forceinline__ double dot(F weight, const double* v0, const double* v1,
                                                 const double* v2) {
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
    double*       ew = D + 2 * kTriPitch; // [12][kTriMax]
    auto issue = [&](const PlaneTile& t, char* slot, int lev) {
        double*      d   = reinterpret_cast<double*>(slot);
        const size_t off = (size_t)lev * Np;
        plane_copy<true>(g, t, d, Mh + off, 0);
        plane_copy<true>(g, t, d + PITCH, Mh + plane + off, 128);
        plane_copy<true>(g, t, d + 2 * PITCH, Mh + 2 * plane + off, 256);
        plane_copy<true>(g, t, d + 3 * PITCH, Wh + off + Np, 384);
    };
    if (threadIdx.x >= kPlaneCols) {
        TriRole<true> r{};
        double        wl[4] = {0, 0, 0, 0}, we[3] = {0, 0, 0}; // Wh at the level's lower interface
        const int     x = (int)threadIdx.x - kPlaneCols;
        auto          seg = [&](const PlaneTile& t, int tile, int l0) {
            r.load(g, t, tile, ew);
            auto below = [&](int slot) {
                const int id = slot < kPlaneCols ? min(t.c0 + slot, g.N - 1)
                                                 : g.phalo[tile * g.phmax + slot - kPlaneCols];
                return Wh[(size_t)l0 * Np + id];
            };
#pragma unroll
            for (int v = 0; v < 4; v++)
                wl[v] = below(r.s[v]);
            if (r.edge)
#pragma unroll
                for (int v = 0; v < 3; v++)
                    we[v] = below(r.e[v]);
        };
        auto comp = [&](const PlaneTile&, const char* slot, int lev, int buf) {
            const double* q      = reinterpret_cast<const double*>(slot);
            const double  rscale = g.lt[kLtRscale * nvi + lev], mdz = -g.lt[kLtRDz * nvi + lev];
            double        m[4][3], dw[4];
            auto          vertex = [&](int sl, double* mv, double& w) { // returns Wh below - above
#pragma unroll
                for (int k = 0; k < 3; k++)
                    mv[k] = q[k * PITCH + sl];
                const double wt = q[3 * PITCH + sl], df = w - wt;
                w               = wt;
                return df;
            };
#pragma unroll
            for (int v = 0; v < 4; v++)
                dw[v] = vertex(r.s[v], m[v], wl[v]);
            double* out = D + buf * kTriPitch;
#pragma unroll
            for (int o = 0; o < 2; o++) {
                const double h = r.dot([&](int k) { return r.w[o][k]; }, m[0], m[1 + o], m[2 + o]);
                const double w = fma(r.a[o][2], dw[2 + o], fma(r.a[o][1], dw[1 + o], r.a[o][0] * dw[0]));
                out[o * kPlaneCols + x] = fma(rscale, h, mdz * w);
            }
            if (r.edge) {
#pragma unroll
                for (int v = 0; v < 3; v++)
                    dw[v] = vertex(r.e[v], m[v], we[v]);
                const double* W = ew + x;
                const double  h = r.dot([&](int k) { return W[k * kTriMax]; }, m[0], m[1], m[2]);
                const double  w = fma(W[11 * kTriMax], dw[2],
                                      fma(W[10 * kTriMax], dw[1], W[9 * kTriMax] * dw[0]));
                out[2 * kPlaneCols + x] = fma(rscale, h, mdz * w);
            }
        };
        role_loop<kStages, kSlotBytes, true>(g, ring, issue, seg, comp);
    }
    else {
        GradRole r{};
        auto     seg  = [&](const PlaneTile& t, int, int) { r.load(g, t); };
        auto     comp = [&](const PlaneTile& t, const char*, int lev, int buf) {
            const double rscale = g.lt[kLtRscale * nvi + lev];
            double       o[3];
            r.apply(D + buf * kTriPitch, o);
            if (t.store)
#pragma unroll
                for (int k = 0; k < 3; k++)
                    divg[k * plane + (size_t)lev * Np + t.c] = (TD)(rscale * o[k]);
        };
        role_loop<kStages, kSlotBytes, false>(g, ring, issue, seg, comp);
    }
}

// Horizontal momentum of a small step: pass 1 of the damping on divg, the pressure gradient, the slow
// tendency; the radial component removed from their sum.
constexpr int kMomStages = 6;
template<class TD>
__global__ void __launch_bounds__(kDivThreads, 1)
    momentum_plane_kernel(Geometry g, Phys P, State s, double dt) {
    extern __shared__ __align__(16) char ring[];
    // a slot: ps (gathered), SlowMh, Mhs (own), then divg (gathered)
    constexpr int kDouble    = PITCH + 6 * kPlaneCols;
    constexpr int kSlotBytes = kDouble * (int)sizeof(double) + 3 * PITCH * (int)sizeof(TD);
    constexpr int kStages    = kMomStages;
    static_assert(kSlotBytes % 16 == 0, "slots keep 16-byte alignment");
    double*      D  = reinterpret_cast<double*>(ring + kStages * kSlotBytes);
    const int    Np = g.Np, nv = g.nv, nvi = g.nvi;
    const size_t plane = (size_t)nv * Np;
    const TD*    divg  = reinterpret_cast<const TD*>(s.divg);
    const bool   damp  = P.DivDampP;
    double*      ew    = D + 2 * kTriPitch; // [9][kTriMax]
    auto issue = [&](const PlaneTile& t, char* slot, int lev) {
        double*      d   = reinterpret_cast<double*>(slot);
        TD*          dg  = reinterpret_cast<TD*>(d + kDouble);
        const size_t off = (size_t)lev * Np;
        plane_copy<true>(g, t, d, s.ps + off, 0);
#pragma unroll
        for (int k = 0; k < 3; k++) {
            plane_copy<false>(g, t, d + PITCH + k * kPlaneCols, s.SlowMh + k * plane + off, 128);
            plane_copy<false>(g, t, d + PITCH + (3 + k) * kPlaneCols, s.Mhs + k * plane + off, 256);
        }
        if (damp)
#pragma unroll
            for (int k = 0; k < 3; k++)
                plane_copy<true>(g, t, dg + k * PITCH, divg + k * plane + off, 384);
    };
    if (threadIdx.x >= kPlaneCols) {
        TriRole<false> r{};
        const int      x    = (int)threadIdx.x - kPlaneCols;
        auto           seg  = [&](const PlaneTile& t, int tile, int) { r.load(g, t, tile, ew); };
        auto           comp = [&](const PlaneTile&, const char* slot, int lev, int buf) {
            if (!damp)
                return;
            const TD* q = reinterpret_cast<const TD*>(reinterpret_cast<const double*>(slot) + kDouble);
            const double rscale = g.lt[kLtRscale * nvi + lev];
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
                out[o * kPlaneCols + x] =
                    rscale * r.dot([&](int k) { return r.w[o][k]; }, m[0], m[1 + o], m[2 + o]);
            if (r.edge) {
#pragma unroll
                for (int v = 0; v < 3; v++)
                    vertex(r.e[v], m[v]);
                const double* W = ew + x;
                out[2 * kPlaneCols + x] =
                    rscale * r.dot([&](int k) { return W[k * kTriMax]; }, m[0], m[1], m[2]);
            }
        };
        role_loop<kStages, kSlotBytes, true>(g, ring, issue, seg, comp);
    }
    else {
        GradRole r{};
        double   gd[7][3] = {}, fr[3] = {};
        auto     seg = [&](const PlaneTile& t, int, int) {
            r.load(g, t);
            const bool valid = t.c < g.N;
#pragma unroll
            for (int j = 0; j < 7; j++) {
                const bool use = valid && (j == 0 || t.point(j) != (int)threadIdx.x); // not a hole
#pragma unroll
                for (int k = 0; k < 3; k++)
                    gd[j][k] = use ? __ldg(g.grad + (size_t)(j * 3 + k) * Np + t.c) : 0.0;
            }
#pragma unroll
            for (int k = 0; k < 3; k++)
                fr[k] = valid ? __ldg(g.func_r + (size_t)k * Np + t.c) : 0.0;
        };
        auto comp = [&](const PlaneTile& t, const char* slot, int lev, int buf) {
            const double* q      = reinterpret_cast<const double*>(slot);
            const double  rscale = g.lt[kLtRscale * nvi + lev];
            double        a[3]   = {0, 0, 0}, l[3] = {0, 0, 0};
#pragma unroll
            for (int j = 0; j < 7; j++) {
                const double pv = q[t.point(j)];
#pragma unroll
                for (int k = 0; k < 3; k++)
                    a[k] = fma(gd[j][k], pv, a[k]);
            }
            if (damp)
                r.apply(D + buf * kTriPitch, l);
            const double* o  = q + PITCH + threadIdx.x;
            const double  kd = g.Kdhz[lev];
            double        T[3];
#pragma unroll
            for (int k = 0; k < 3; k++)
                T[k] = fma(-rscale, fma(kd, l[k], a[k]), o[k * kPlaneCols]) * dt;
            const double vr = T[0] * fr[0] + T[1] * fr[1] + T[2] * fr[2];
            if (t.store)
#pragma unroll
                for (int k = 0; k < 3; k++)
                    s.Mhs[k * plane + (size_t)lev * Np + t.c] =
                        o[(3 + k) * kPlaneCols] + fma(-vr, fr[k], T[k]);
        };
        role_loop<kStages, kSlotBytes, false>(g, ring, issue, seg, comp);
    }
}

template<class TD>
void launch_divm0_t(const Geometry& g, const Phys& P, const double* M, const double* W, double* divg,
                    cudaStream_t st) {
    constexpr size_t smem = sizeof(double) * (kDiv0Stages * 4 * PITCH + 2 * kTriPitch + 12 * kTriMax);
    static SmemOptIn opt;
    if (opt.ensure(divm0_plane_kernel<TD>, smem) == cudaSuccess)
        divm0_plane_kernel<TD><<<plane_ctas(g, 1), kDivThreads, smem, st>>>(
            g, P, M, W, reinterpret_cast<TD*>(divg));
}
template<class TD>
void launch_momentum_t(const Geometry& g, const Phys& P, const State& s, double dt,
                       cudaStream_t st) {
    constexpr size_t smem = kMomStages * (sizeof(double) * (PITCH + 6 * kPlaneCols) + sizeof(TD) * 3 * PITCH)
                            + sizeof(double) * (2 * kTriPitch + 9 * kTriMax);
    static SmemOptIn opt;
    if (opt.ensure(momentum_plane_kernel<TD>, smem) == cudaSuccess)
        momentum_plane_kernel<TD><<<plane_ctas(g, 1), kDivThreads, smem, st>>>(g, P, s, dt);
}

// ---------------------------------------------------------------------------------------------
// Advection and Coriolis of an RK stage (Compute_Advec_Cori1 / _Poles, Compute_Advec_Cori2,
// src/headers/dyn/thor_adv_cor.h:51-536). The cartesian velocity v = M / rho + (w / rho) r^ of a column
// is formed once per level in shared memory (own columns and halo), where the column-tile form formed
// it at each of the seven points; the flux divergence is sum_j v_j (div_j . M_j). The velocities run
// one level ahead, so that the vertical flux has the level above at hand.
// ---------------------------------------------------------------------------------------------
constexpr int kAdvStages = 5, kAdvSlot = 5 * PITCH + kPlaneCols;
__global__ void __launch_bounds__(kPlaneCols, 2) adv_plane_kernel(Geometry g, Phys P, State s) {
    extern __shared__ __align__(16) double ringd[];
    double*      sv = ringd + kAdvStages * kAdvSlot; // [2][3][PITCH]
    const int    Np = g.Np, nv = g.nv, nvi = g.nvi, x = threadIdx.x;
    const size_t plane = (size_t)nv * Np;
    const double* lt   = g.lt;
    const double  Omega = P.Omega;
    double        d[7][3], fr[3], frh[3], vprev[3], vcur[3], vnext[3], whl = 0.0;
    const double* const src[6] = {s.Mhk, s.Mhk + plane, s.Mhk + 2 * plane, s.Rhok, s.Wk, s.Whk + Np};
    auto issue = [&](const PlaneTile& t, double* slot, int lev) {
        plane_issue<5, 1, PITCH>(g, t, slot, src, lev);
    };
    auto vel = [&](double m0, double m1, double m2, double rho, double w, const double* f, double* v) {
        const double yr = 1.0 / rho, wr = div_rcp(w, rho, yr);
        v[0] = fma(wr, f[0], div_rcp(m0, rho, yr));
        v[1] = fma(wr, f[1], div_rcp(m1, rho, yr));
        v[2] = fma(wr, f[2], div_rcp(m2, rho, yr));
    };
    auto seg = [&](const PlaneTile& t, int l0) {
        const bool valid = t.c < g.N;
        const int  c     = min(t.c, g.N - 1);
#pragma unroll
        for (int j = 0; j < 7; j++) {
            const bool use = valid && (j == 0 || t.point(j) != x); // not a hole
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
        vel(b[x], b[PITCH + x], b[2 * PITCH + x], b[3 * PITCH + x], b[4 * PITCH + x], fr, vnext);
#pragma unroll
        for (int k = 0; k < 3; k++)
            v[k * PITCH + x] = vnext[k];
        if (t.hid >= 0) {
            const double* h = b + kPlaneCols + x;
            double        vh[3];
            vel(h[0], h[PITCH], h[2 * PITCH], h[3 * PITCH], h[4 * PITCH], frh, vh);
#pragma unroll
            for (int k = 0; k < 3; k++)
                v[k * PITCH + kPlaneCols + x] = vh[k];
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
            const double rscale = lt[kLtRscale * nvi + lev], rho = b[3 * PITCH + x];
            double       r2p = 1.0, r2m = 1.0, r2l = 1.0, C[3];
            if (P.DeepModel) {
                r2p  = lt[kLtR2hD * nvi + lev + 1];
                r2m  = lt[kLtR2cD * nvi + lev];
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
            (void)r2m;
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
    lag_loop<kAdvStages, kAdvSlot, true>(g, ringd, issue, seg, prep, comp);
}

// ---------------------------------------------------------------------------------------------
// A hyperdiffusion pass (Diffusion_Op + Diffusion_Op_Poles, src/headers/dyn/thor_diff.h:54-880, and
// Correct_Horizontal, :882-915, on the last): the Laplacian's 7 weights per column stay in registers
// and serve the six variables. kFirst: the arguments rho, v, w, Rd T (or Cv T) are formed once per
// column in the ring (own columns and halo), where each of the seven points formed them before. The
// pass before the last stores its result times rho for v, w and T, which is the last one's argument.
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
    auto issue = [&](const PlaneTile& t, double* slot, int lev) {
        plane_issue<6, 0, PITCH>(g, t, slot, src, lev);
    };
    auto seg = [&](const PlaneTile& t, int) {
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
                convert(b + x, t.c);
            if (t.hid >= 0)
                convert(b + kPlaneCols + x, t.hid);
        }
    };
    auto comp = [&](const PlaneTile& t, const double* b, int lev, int) {
        double a0[6], acc[6];
#pragma unroll
        for (int v = 0; v < 6; v++) {
            a0[v]  = b[v * PITCH + x];
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
        const double r = fr[0] * acc[1] + fr[1] * acc[2] + fr[2] * acc[3];
        s.diffrh[i]    = acc[0];
#pragma unroll
        for (int k = 0; k < 3; k++)
            s.diffmh[k * plane + i] = fma(-fr[k], r, acc[1 + k]);
        s.diffw[i]  = acc[4];
        s.diffpr[i] = acc[5];
    };
    lag_loop<kDiffStages, kDiffSlot, false>(g, ringd, issue, seg, prep, comp);
}

template<bool kFirst, bool kUni>
void launch_diffusion_t(const Geometry& g, const Phys& P, const State& s, const double* in, double* out,
                        bool last, bool scale, cudaStream_t st) {
    constexpr size_t smem = sizeof(double) * kDiffStages * kDiffSlot;
    static SmemOptIn opt;
    if (opt.ensure(diffusion_plane_kernel<kFirst, kUni>, smem) == cudaSuccess)
        diffusion_plane_kernel<kFirst, kUni>
            <<<plane_ctas(g, 2), kPlaneCols, smem, st>>>(g, P, s, in, out, last, scale);
}

} // namespace

void launch_adv_planes(const Geometry& g, const Phys& P, const State& s, cudaStream_t st) {
    constexpr size_t smem = sizeof(double) * (kAdvStages * kAdvSlot + 6 * PITCH);
    static SmemOptIn opt;
    if (opt.ensure(adv_plane_kernel, smem) == cudaSuccess)
        adv_plane_kernel<<<plane_ctas(g, 2), kPlaneCols, smem, st>>>(g, P, s);
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
void launch_momentum_planes(const Geometry& g, const Phys& P, const State& s, double dt,
                            cudaStream_t st) {
    if (P.mixed && kDivgF32)
        launch_momentum_t<float>(g, P, s, dt, st);
    else
        launch_momentum_t<double>(g, P, s, dt, st);
}

void launch_tri_weights(const Geometry& g, const int* ev, int tiles, double* tw, double* gw, double* ew,
                        cudaStream_t st) {
    tri_weights_kernel<<<(g.N + 127) / 128, 128, 0, st>>>(g, tw, gw);
    edge_weights_kernel<<<tiles, kTriMax, 0, st>>>(g, ev, g.ptri_n, tiles, ew);
}

} // namespace thorx
