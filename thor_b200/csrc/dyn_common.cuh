// Device helpers shared by the dynamical-core kernels.
#pragma once

#include <mutex>

#include "thorx_internal.h"

namespace thorx {

// Gas constant and heat capacity of a cell. kUni (Phys::uniform_thermo: every cell's Rd and Cp
// are Phys::Rd and Phys::Cp, which the context checks whenever the fields are set): the scalars, so
// the compiler folds the expressions built from them (Rd / (Cp - Rd) and the like) into per-thread
// constants; they are the same values, so the results are the same bits as the per-cell loads.
template<bool kUni> __device__ __forceinline__ double rd_at(const Phys& P, const State& s, int i) {
    if constexpr (kUni)
        return P.Rd;
    else
        return s.Rd[i];
}
template<bool kUni> __device__ __forceinline__ double cp_at(const Phys& P, const State& s, int i) {
    if constexpr (kUni)
        return P.Cp;
    else
        return s.Cp[i];
}

// a / b rounded to nearest, from y = 1/b rounded to nearest, with fused multiply-adds only.
// Markstein's theorem (P. W. Markstein, IBM J. Res. Develop. 34(1):111-119, 1990; J.-M. Muller et
// al., Handbook of Floating-Point Arithmetic, 2nd ed., 2018, sect. 4.7): if y = RN(1/b) and q is
// within one ulp of a/b, the remainder a - b q is exact in one fma and RN(q + (a - b q) y) =
// RN(a/b). q0 = RN(a y) is only within 1.5 ulp, so one correction step comes first. The result is
// the IEEE quotient a / b bit for bit while a, b, the quotient and the remainders are normal
// numbers (every field and grid quantity divided here); a zero numerator returns RN(a y), the
// signed zero a / b has. Used where one divisor (a cell's sub-triangle area) serves many divisions,
// so the one IEEE division of the reciprocal is paid once per column.
__device__ __forceinline__ double div_rcp(double a, double b, double y) {
    const double q0 = __dmul_rn(a, y);
    const double q1 = __fma_rn(__fma_rn(-q0, b, a), y, q0);
    const double q2 = __fma_rn(__fma_rn(-q1, b, a), y, q1);
    return a == 0.0 ? q0 : q2;
}
__device__ __forceinline__ float div_rcp(float a, float b, float y) {
    const float q0 = __fmul_rn(a, y);
    const float q1 = __fmaf_rn(__fmaf_rn(-q0, b, a), y, q0);
    const float q2 = __fmaf_rn(__fmaf_rn(-q1, b, a), y, q1);
    return a == 0.0f ? q0 : q2;
}

// The largest dynamic shared memory a kernel has been opened to, per device (the attribute is a
// per-device setting; a process may hold contexts on several devices, and host threads may launch
// concurrently). A size is recorded only once the driver has accepted it; a refusal is returned
// (and stays the runtime's last error, which the caller's error check reports), and the next
// launch asks again.
constexpr int kMaxDevices = 64;
struct SmemOptIn {
    std::mutex mu;
    size_t     bytes[kMaxDevices] = {};
    template<class Kernel>
    cudaError_t ensure(Kernel* kernel, size_t smem) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess)
            dev = -1;
        std::lock_guard<std::mutex> lock(mu);
        if (dev >= 0 && dev < kMaxDevices && smem <= bytes[dev])
            return cudaSuccess;
        const cudaError_t e =
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess && dev >= 0 && dev < kMaxDevices)
            bytes[dev] = smem;
        return e;
    }
};

// Programmatic dependent launch: a kernel of the step may start while the one before it in the stream
// still runs, as far as its CTAs find room, and loads what no kernel writes (tables, weights) before
// step_wait(), which returns when everything before it in the stream is complete and visible. Every
// kernel launched this way calls step_begin() first and step_wait() before it touches a field, so the
// order of the step is transitive; a kernel launched the ordinary way waits for all of them. glevel 4, 32
// levels: the step 551 -> 478 us; glevel 5, 37 levels: 1143 -> 1043; glevel 6, 48 levels: 4187 -> 4133.
__device__ __forceinline__ void step_begin() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void step_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template<class... P, class... A>
inline cudaError_t launch_step(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                               A... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim          = grid;
    cfg.blockDim         = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream           = st;
    cfg.attrs            = &at;
    cfg.numAttrs         = 1;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

} // namespace thorx
