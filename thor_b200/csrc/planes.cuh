// Level planes of a tile of 256 columns staged through shared memory for the horizontal stencils.
//
// A tile is 256 consecutive columns (one 16 x 16 rhombus of the grid); its halo is the neighbours
// outside it (at most 66 columns for rhombi of 16 x 16, Geometry::phalo). Per level a kernel copies
// the planes its stencil gathers (own columns and halo) and those it reads at the column only into
// one slot of a shared-memory ring by cp.async, kStages - 1 levels ahead of the computation (kStages - 2
// in the loops that prepare a level before they use it); one
// thread then computes one column, its stencil points being slots of the ring (Geometry::pnb), its
// operator weights staying in registers from level to level.
//
// Why this form: a warp's global gather of a stencil point touches three to four cache lines (the
// rows of a rhombus are 16 columns, shifted by one, with the ends in other rhombi), so kernels that
// gather from global memory are limited by L1 tag lookups and by the latency of the few loads that
// registers let a warp keep in flight; from shared memory a point costs two wavefronts, and the
// copies in flight cost no registers. The work is the (tile, level) pairs in tile order, divided
// evenly over as many CTAs as are resident, so that no last wave is nearly empty and a grid of few
// tiles still fills the chip; a CTA reloads its weights only where its range enters another tile.
#pragma once

#include <cstdint>

#include "dyn_common.cuh"

namespace thorx {

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async8(double* dst, const double* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
    asm volatile("cp.async.commit_group;" ::: "memory");
}
template<int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Slots of a gathered plane. Rhombi of 16 x 16: an 18 x 18 picture of the tile and its halo with rows
// kRowPitch apart (a row's own columns start on a 16-byte boundary), so that the 16 columns of a row
// read any stencil point from consecutive 8-byte words: no bank conflicts (with the halo behind the
// tile's columns, the row ends hit an occupied bank and every point took four wavefronts for two). Other
// grids: the tile's columns in order, then the halo.
template<int PITCH> __device__ __forceinline__ int own_slot(int x) {
    return PITCH == kPitchRhombus ? plane_slot(x & 15, x >> 4) : x;
}

// One thread's view of the tile it works on.
struct PlaneTile {
    int      c0, c;    // first column of the tile; this thread's column (threads 0..255)
    int      ncopy;    // own columns that exist (a multiple of 32)
    int      nh;       // halo columns
    int      hid;      // the halo column thread threadIdx.x copies (-1: none) and its slot
    int      hslot;
    int      own;      // slot of the thread's column
    bool     store;    // the column is this context's to compute and store
    unsigned nb[3];    // slots of the stencil points pt1..pt6, two per word
    __device__ __forceinline__ int point(int j) const { // slot of point j = 0..6
        return j == 0 ? own : (int)((nb[(j - 1) >> 1] >> (16 * ((j - 1) & 1))) & 0xffffu);
    }
};

// X0: the first of the 256 threads that hold the tile's columns in order.
template<int PITCH, int X0 = 0>
__device__ __forceinline__ PlaneTile plane_tile(const Geometry& g, int tile) {
    PlaneTile t;
    const int x = (int)threadIdx.x - X0;
    t.c0    = tile * kPlaneCols;
    t.ncopy = min(kPlaneCols, g.Np - t.c0);
    t.c     = t.c0 + x;
    t.nh    = g.pnhalo[tile];
    t.hid   = x < t.nh ? g.phalo[tile * g.phmax + x] : -1;
    t.hslot = x < t.nh ? g.phslot[tile * g.phmax + x] : 0;
    t.own   = own_slot<PITCH>(x & (kPlaneCols - 1));
    t.store = x < kPlaneCols && t.c >= g.tile0 * kTileCols && t.c < g.col_end;
    const bool valid = x < kPlaneCols && t.c < g.N;
#pragma unroll
    for (int k = 0; k < 3; k++)
        t.nb[k] = valid ? g.pnb[k * g.Np + t.c] : (unsigned)t.own * 0x10001u;
    return t;
}

// Copies one level of NG gathered planes and NO own planes into a ring slot (thread groups of 128
// take alternate planes; every thread below nh takes one halo column).
template<int NG, int NO, int PITCH>
__device__ __forceinline__ void plane_issue(const Geometry& g, const PlaneTile& t, double* slot,
                                            const double* const (&src)[NG + NO], int lev) {
    const int    x = threadIdx.x, grp = x >> 7, y = (x & 127) * 2, ys = own_slot<PITCH>(y);
    const size_t off = (size_t)lev * g.Np;
    if (x < kPlaneCols && y < t.ncopy) {
#pragma unroll
        for (int p = 0; p < NG + NO; p++)
            if ((p & 1) == grp) {
                double* d = p < NG ? slot + p * PITCH + ys : slot + NG * PITCH + (p - NG) * kPlaneCols + y;
                cp_async16(d, src[p] + off + t.c0 + y);
            }
    }
    if (t.hid >= 0) {
#pragma unroll
        for (int p = 0; p < NG; p++)
            cp_async8(slot + p * PITCH + t.hslot, src[p] + off + t.hid);
    }
    if constexpr (PITCH != kPitchRhombus) // more halo columns than threads
        for (int k = x + blockDim.x; k < t.nh; k += blockDim.x) {
            const int e = (t.c0 / kPlaneCols) * g.phmax + k;
#pragma unroll
            for (int p = 0; p < NG; p++)
                cp_async8(slot + p * PITCH + g.phslot[e], src[p] + off + g.phalo[e]);
        }
}

// Runs this CTA's share of the (tile, level) pairs: seg(tile view) where the range enters a tile,
// then comp(slot, level) for each level with the level's planes in the slot.
template<int NG, int NO, int PITCH, int kStages, class Seg, class Comp>
__device__ __forceinline__ void plane_loop(const Geometry& g, double* ring,
                                           const double* const (&src)[NG + NO], Seg seg,
                                           Comp comp) {
    constexpr int   kSlot = NG * PITCH + NO * kPlaneCols;
    const int       t0 = g.tile0 * kTileCols / kPlaneCols;
    const int       t1 = (g.col_end + kPlaneCols - 1) / kPlaneCols;
    const int       nv = g.nv;
    const long long total = (long long)(t1 - t0) * nv;
    int             u     = (int)(total * blockIdx.x / gridDim.x);
    const int       u1    = (int)(total * (blockIdx.x + 1) / gridDim.x);
    bool            first = true;
    step_begin();
    while (u < u1) {
        const int tile = t0 + u / nv, l0 = u % nv, n = min(nv - l0, u1 - u);
        const PlaneTile t = plane_tile<PITCH>(g, tile);
        seg(t);
        if (first) // the tables and weights above are nobody's to write
            step_wait();
        first = false;
#pragma unroll
        for (int k = 0; k < kStages - 1; k++) {
            if (k < n)
                plane_issue<NG, NO, PITCH>(g, t, ring + k * kSlot, src, l0 + k);
            cp_async_commit();
        }
        int slot = 0;
        for (int i = 0; i < n; i++) {
            cp_async_wait<kStages - 2>();
            __syncthreads(); // the level's copies are visible; the previous level's slot is read
            const int ns = slot == 0 ? kStages - 1 : slot - 1;
            if (i + kStages - 1 < n)
                plane_issue<NG, NO, PITCH>(g, t, ring + ns * kSlot, src, l0 + i + kStages - 1);
            cp_async_commit();
            comp(t, ring + slot * kSlot, l0 + i);
            slot = slot + 1 == kStages ? 0 : slot + 1;
        }
        cp_async_wait<0>();
        __syncthreads(); // every slot read before the next tile's copies
        u += n;
    }
}

// The same ring with a preparation one level ahead: iteration i waits for level i, then prep(slot,
// level i) works on the slot (each thread on its own entries) while comp(slot, level i - 1) reads the
// slot prepared before; one barrier a level. kAhead: prep also runs on the level above the range. seg
// loads what belongs to the grid, below what the range's first level needs of the fields below it.
template<int NG, int NO, int kStages, bool kAhead, class Seg, class Below, class Prep, class Comp>
__device__ __forceinline__ void lag_loop(const Geometry& g, double* ring,
                                         const double* const (&src)[NG + NO], Seg seg, Below below,
                                         Prep prep, Comp comp) {
    constexpr int   kSlotDoubles = NG * kPitchRhombus + NO * kPlaneCols;
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
        const int       np   = kAhead && l0 + n < nv ? n + 1 : n; // levels prepared
        const PlaneTile t    = plane_tile<kPitchRhombus>(g, tile);
        seg(t);
        if (first) // the tables and weights above are nobody's to write
            step_wait();
        first = false;
#pragma unroll
        for (int k = 0; k < kStages - 2; k++) {
            if (k < np)
                plane_issue<NG, NO, kPitchRhombus>(g, t, ring + k * kSlotDoubles, src, l0 + k);
            cp_async_commit();
        }
        below(t, l0);
        int cur = 0, prev = kStages - 1, next = kStages - 2;
        for (int i = 0; i <= n; i++) {
            cp_async_wait<kStages - 3>();
            __syncthreads(); // level i is copied, level i - 1 prepared, slot `next` read
            if (i + kStages - 2 < np)
                plane_issue<NG, NO, kPitchRhombus>(g, t, ring + next * kSlotDoubles, src,
                                                   l0 + i + kStages - 2);
            cp_async_commit();
            if (i < np)
                prep(t, ring + cur * kSlotDoubles, l0 + i, i & 1);
            if (i > 0)
                comp(t, ring + prev * kSlotDoubles, l0 + i - 1, (i - 1) & 1);
            prev = cur;
            cur  = cur + 1 == kStages ? 0 : cur + 1;
            next = next + 1 == kStages ? 0 : next + 1;
        }
        cp_async_wait<0>();
        __syncthreads();
        u += n;
    }
}

// Shared memory of a ring, and the CTAs that share its work: those resident, at least one level each.
template<int NG, int NO, int PITCH, int kStages>
constexpr size_t plane_ring_bytes() {
    return sizeof(double) * kStages * (NG * PITCH + NO * kPlaneCols);
}
inline int plane_ctas(const Geometry& g, int per_sm) {
    const int t0 = g.tile0 * kTileCols / kPlaneCols;
    const int t1 = (g.col_end + kPlaneCols - 1) / kPlaneCols;
    const long long total = (long long)(t1 - t0) * g.nv, most = (long long)g.nsm * per_sm;
    return (int)(total < most ? total : most);
}

} // namespace thorx
