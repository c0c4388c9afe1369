// demag_inst.cuh -- device helpers shared by the demag passes: the scaled
// magnetisation and the per-instance views of PassArgs.
#pragma once
#include "demag.cuh"

namespace umag {

static constexpr double kMu0f = 4 * 3.1415926535897932384626433 * 1e-7;  // clh/constants.clh:5

// copypadmul2.cl:13-20: MU0*Ms (FP64 product rounded to float32) * vol * m
__device__ __forceinline__ float scaled_m(const PassArgs& a, const float* m, int i, float msmul) {
    float fac = a.Ms == nullptr ? msmul : __fmul_rn(msmul, __ldg(a.Ms + i));
    float bsat = (float)(kMu0f * (double)fac);
    float w = a.vol == nullptr ? 1.0f : __fmul_rn(1.0f, __ldg(a.vol + i));
    return __fmul_rn(__fmul_rn(bsat, w), m[i]);
}

// Per-instance views of PassArgs for batched launches (an ensemble of
// same-size instances, instance ib): spectrum scratch, field output, the
// instance's controller fields (m slots, active flag) and its Ms.  With
// ib = 0 (single-instance kernels) every offset folds away.
__device__ __forceinline__ float2* inst_spec(const PassArgs& a, int ib) { return a.spec + (long)ib * a.spec_stride; }
__device__ __forceinline__ float* inst_B(const PassArgs& a, int ib, int c) { return a.B[c] + (long)ib * a.b_stride; }
__device__ __forceinline__ bool inst_inactive(const PassArgs& a, int ib) {
    if (!a.active) return false;
    return !*reinterpret_cast<const int*>(reinterpret_cast<const char*>(a.active) + (long)ib * a.ctl_stride);
}
__device__ __forceinline__ const float* inst_m(const PassArgs& a, int ib, int c) {
    if (!a.m_ind) return a.m[c];
    const char* slot = reinterpret_cast<const char*>(a.m_sel ? a.m_ind_w : a.m_ind) + (long)ib * a.ctl_stride;
    return *reinterpret_cast<float* const*>(slot) + (long)c * a.ncell;
}
__device__ __forceinline__ float inst_msmul(const PassArgs& a, int ib) { return a.ms_mul_b ? a.ms_mul_b[ib] : a.Ms_mul; }

// record a pass that gave up waiting for a bulk copy: the counter, and the
// instance's controller status (7, as the torque kernel's tile wait) when
// the launch belongs to a simulation
__device__ __forceinline__ void pass_timeout(const PassArgs& a, int ib) {
    atomicAdd(a.timeouts, 1u);
    if (a.fault) atomicCAS(reinterpret_cast<int*>(reinterpret_cast<char*>(a.fault) + (long)ib * a.ctl_stride), 0, 7);
}

// Spectrum: 4-column blocks [c][kz][kx/4][y][kx%4].  Offset of column kx, row y.
__device__ __forceinline__ long spec_at(int Ny, int kx, int y) { return ((long)(kx >> 2) * Ny + y) * 4 + (kx & 3); }
// Kernel spectrum element (kz, ky, kx), kz and ky in the stored non-redundant
// block: 4-column blocks [kz][kx/4][ky][kx%4], or rows of pitch Kp (caller-owned)
__device__ __forceinline__ long kern_idx(const PassArgs& a, int kz, int ky, int kx, int hy) {
    return a.Kblocked ? (((long)kz * (a.Kp >> 2) + (kx >> 2)) * hy + ky) * 4 + (kx & 3)
                      : ((long)kz * hy + ky) * a.Kp + kx;
}

// cp.async (global -> shared, asynchronous)
__device__ __forceinline__ void cpa4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src));
}
__device__ __forceinline__ void cpa8(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cpa_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

}  // namespace umag
