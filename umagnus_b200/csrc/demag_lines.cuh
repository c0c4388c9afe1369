// demag_lines.cuh -- the demag passes on line transforms (fft_line.cuh).
//
//   X  (4 rows y of one component and plane z): scale m by MU0*Ms*vol, real-
//      to-complex transform along x -> spectrum
//   Z  (one column): transform along z, in registers, in place
//   Y  (4 columns kx of one plane kz, all components): forward along y, 3x3
//      symmetric kernel multiply, inverse; rows y < Ny back
// and the inverses Z^-1, X^-1 (crop, B overwritten).  Meshes of one layer
// have no Z.  The padded sizes are this file's choice: the shortest
// supported lengths that hold the mesh (any padding of at least 2N - 1
// gives the same convolution), so sizes without a plan of their own run on
// the next longer one.
//
// Spectrum layout: [c][kz][kx/4][y][kx%4]: Y reads and writes contiguous runs
// of 32 Ny bytes, X whole 128-byte lines (4 columns x 4 rows).
#pragma once
#include "demag_inst.cuh"
#include "fft_line.cuh"
#include "tile.cuh"

namespace umag {

// row pitch or line stride of at least n slots, = r (mod 16)
constexpr int pitch16(int n, int r) { return n + ((r - n) % 16 + 16) % 16; }

// asynchronous (the loads that follow do not wait for it): cpa_wait_all and a
// barrier come before its use
__device__ __forceinline__ void tw_copy(float2* dst, const float2* __restrict__ src, int n, int tid, int nth) {
    for (int i = tid; i < n; i += nth) cpa8(dst + i, src + i);
}

// ================================================================ X
// lanes: parity fastest, then the T threads of a row, then the 4 rows
template <int L, int NPAR> struct XShape {
    using LN = Line<L>;
    static constexpr int M = NPAR * L, T = LN::T, NT = 4 * NPAR * T;
    static constexpr int SP = pitch16(LN::slots, 8);              // parity lines
    static constexpr int SR = NPAR * SP + (T < 8 ? 4 : 0);       // rows
    static constexpr int ZP = pitch16(M + 1, 4);                  // half-spectrum rows
    static constexpr int WR = M / 2 + 1;                          // exp(-2 pi i k / 2M), k <= M/2
    // the rows and the exchange lines share their room
    static constexpr size_t smem = sizeof(float2) * ((size_t)M + WR + 4 * (SR > ZP ? SR : ZP));
    // forward: values, scales and addresses
    static constexpr int regs = (LN::NE <= 8 ? 64 : LN::NE <= 12 ? 80 : 96) + (NPAR == 1 ? 32 : 0);
    static constexpr int minb0 = 65536 / (regs * ((NT + 31) / 32 * 32)), minb1 = (int)(227 * 1024 / (smem + 1024));
    static constexpr int minb = minb0 < minb1 ? (minb0 < 16 ? minb0 : 16) : (minb1 < 16 ? minb1 : 16);
};

// Forward: z[n] = x[2n] + i x[2n+1] of every row (zero above Nx), transform of
// length M = NPAR L, X[k] = E + W^k O for k = 0..M.
// Four rows a CTA: stores of whole 128-byte lines, and CTAs enough on small
// meshes.  Up to some 100,000 cells the time is the latency of one CTA (the
// controller read, the rows, one exchange, the unpack), above it the spectrum
// stores.  64x64: 3.1 us, 250x250 with a geometry map: 5.0 us (the
// runtime-planned pass took 45.7), 1024x1024: 25.1 us (30.6).  Large meshes with
// an Ms map are bound by latency at the CTAs that fit: with rows and exchange
// lines in one room, a register cap, and each parity scaling half of the values that both
// need, RK45DP on 512x512x32 with regions takes 7479 us a step (7771 before).
template <int L, int NPAR>
__global__ void __launch_bounds__(4 * NPAR * Line<L>::T, XShape<L, NPAR>::minb) k_x_fwd(const __grid_constant__ PassArgs a) {
    using S = XShape<L, NPAR>;
    using LN = typename S::LN;
    constexpr int M = S::M, T = S::T, NT = S::NT;
    extern __shared__ __align__(16) float2 sm[];
    float2 *tw = sm, *twr = tw + M, *ex = twr + S::WR, *Zs = ex;
    const int ib = blockIdx.z;
    const int tid = threadIdx.x, p = tid % NPAR, t = (tid / NPAR) % T, row = tid / (NPAR * T);
    const int c = blockIdx.y / a.Nz, z = blockIdx.y - c * a.Nz, y0 = blockIdx.x * 4, y = y0 + row, Nx = a.Nx;
    tw_copy(tw, a.fx.tw, M, tid, NT);
    tw_copy(twr, a.twr, S::WR, tid, NT);
    const float* m = nullptr;
    bool off = false;
    if (a.early) {
        m = inst_m(a, ib, c);
        off = inst_inactive(a, ib);
    }
    pdl_wait();
    pdl_trigger();
    if (!a.early) {
        m = inst_m(a, ib, c);
        off = inst_inactive(a, ib);
    }
    if (off) {
        cpa_wait_all();
        return;
    }
    const float msm = inst_msmul(a, ib);
    P2 v[1][LN::NE];
    {
        // every load is issued before the first is used: cells outside the
        // mesh read a cell inside and become zero afterwards
        const int i0 = (z * a.Ny + min(y, a.Ny - 1)) * Nx;
        // pairs (x, x+1) in one 8-byte load where the rows start on 8 bytes
        const bool uni = a.Ms == nullptr && a.vol == nullptr;
        const bool pairs = (Nx & 1) == 0 && (reinterpret_cast<uintptr_t>(m) & 7) == 0;
        constexpr int NV = LN::Q1 * LN::R1;
        float2 f[NV];
        auto xof = [&](int i) { return 2 * (t + T * (i / LN::R1) + LN::B1 * (i % LN::R1)); };
        if (pairs) {
#pragma unroll
            for (int i = 0; i < NV; i++) f[i] = *reinterpret_cast<const float2*>(m + i0 + min(xof(i), Nx - 2));
        } else {
#pragma unroll
            for (int i = 0; i < NV; i++)
                f[i] = make_float2(m[i0 + min(xof(i), Nx - 1)], m[i0 + min(xof(i) + 1, Nx - 1)]);
        }
        if (uni) {
            const float bsat = (float)(kMu0f * (double)msm);  // scaled_m's rounding: (bsat * 1) * m = bsat * m
#pragma unroll
            for (int i = 0; i < NV; i++) f[i] = make_float2(__fmul_rn(bsat, f[i].x), __fmul_rn(bsat, f[i].y));
        } else {
            // the two parities of a row need the same values: each scales half of them
            constexpr int NS = (NV + NPAR - 1) / NPAR;
            float2 bs[NS], g[NS];
            int x0[NS], x1[NS];
#pragma unroll
            for (int i = 0; i < NS; i++) {
                const bool odd = NPAR == 2 && p && 2 * i + 1 < NV;
                const int x = odd ? xof(NPAR * i + 1) : xof(NPAR * i);
                x0[i] = i0 + min(x, Nx - 1);
                x1[i] = i0 + min(x + 1, Nx - 1);
                g[i] = odd ? f[NPAR * i + 1 < NV ? NPAR * i + 1 : 0] : f[NPAR * i];
                bs[i] = a.Ms ? make_float2(__ldg(a.Ms + x0[i]), __ldg(a.Ms + x1[i])) : make_float2(1.f, 1.f);
            }
#pragma unroll
            for (int i = 0; i < NS; i++)  // MU0*Ms: FP64 product rounded to float32 (copypadmul2.cl:13-20)
                bs[i] = make_float2((float)(kMu0f * (double)(a.Ms ? __fmul_rn(msm, bs[i].x) : msm)),
                                    (float)(kMu0f * (double)(a.Ms ? __fmul_rn(msm, bs[i].y) : msm)));
            if (a.vol) {
                float2 w[NS];
#pragma unroll
                for (int i = 0; i < NS; i++) w[i] = make_float2(__ldg(a.vol + x0[i]), __ldg(a.vol + x1[i]));
#pragma unroll
                for (int i = 0; i < NS; i++) bs[i] = make_float2(__fmul_rn(bs[i].x, w[i].x), __fmul_rn(bs[i].y, w[i].y));
            }
#pragma unroll
            for (int i = 0; i < NS; i++) {
                g[i] = make_float2(__fmul_rn(bs[i].x, g[i].x), __fmul_rn(bs[i].y, g[i].y));
                if constexpr (NPAR == 2) {
                    const float2 o = make_float2(__shfl_xor_sync(0xffffffffu, g[i].x, 1),
                                                 __shfl_xor_sync(0xffffffffu, g[i].y, 1));
                    f[2 * i] = p ? o : g[i];
                    if (2 * i + 1 < NV) f[2 * i + 1 < NV ? 2 * i + 1 : 0] = p ? g[i] : o;
                } else {
                    f[i] = g[i];
                }
            }
        }
#pragma unroll
        for (int i = 0; i < NV; i++) {
            const int x = xof(i), b = t + T * (i / LN::R1);
            const bool in = y < a.Ny && (LN::B1 % T == 0 || b < LN::B1);
            v[0][i] = p2(in && x < Nx ? f[i].x : 0.f, in && x + 1 < Nx ? f[i].y : 0.f);
        }
    }
    cpa_wait_all();
    __syncthreads();
    line_fwd<LN, NPAR, 1, 1>(v, t, p, ex + row * S::SR + p * S::SP, 0, tw);
    __syncthreads();  // the exchange lines become rows
#pragma unroll
    for (int q = 0; q < LN::Qf; q++) {
        const int b = t + T * q;
        if (LN::Bf % T == 0 || b < LN::Bf)
#pragma unroll
            for (int k = 0; k < LN::Rf; k++) Zs[row * S::ZP + NPAR * LN::freq(b, k) + p] = f2(v[0][q * LN::Rf + k]);
    }
    __syncthreads();
    // X[k] = E + W^k O, X[M-k] = conj(E - W^k O); lanes: 4 columns x 4 rows
    float2* out = inst_spec(a, ib) + ((long)c * a.Pz + z) * a.Ny * a.Lx;
#pragma unroll 4
    for (int e = tid; e < (M / 8 + 1) * 16; e += NT) {
        const int k = (e >> 4) * 4 + (e & 3), r = (e >> 2) & 3;
        if (k > M / 2 || y0 + r >= a.Ny) continue;
        const float2 A = Zs[r * S::ZP + k], B = Zs[r * S::ZP + (k == 0 ? 0 : M - k)];
        const float2 E = make_float2(0.5f * (A.x + B.x), 0.5f * (A.y - B.y));
        const float2 D = make_float2(0.5f * (A.x - B.x), 0.5f * (A.y + B.y));
        const float2 O = make_float2(D.y, -D.x), W = twr[k];
        const float2 WO = make_float2(fma_rn(W.x, O.x, -mul_rn(W.y, O.y)), fma_rn(W.x, O.y, mul_rn(W.y, O.x)));
        out[spec_at(a.Ny, k, y0 + r)] = make_float2(E.x + WO.x, E.y + WO.y);
        if (2 * k != M) out[spec_at(a.Ny, M - k, y0 + r)] = make_float2(E.x - WO.x, WO.y - E.y);
    }
}

// Inverse: Z[k] = (X[k] + conj X[M-k]) + i conj(W^k) (X[k] - conj X[M-k]) of
// every row, inverse transform, x < Nx to B.  250x250: 4.1 us (the
// runtime-planned pass took 45.7), 1024x1024: 26.1 us (30.0).
template <int L, int NPAR>
__global__ void __launch_bounds__(4 * NPAR * Line<L>::T) k_x_inv(const __grid_constant__ PassArgs a) {
    using S = XShape<L, NPAR>;
    using LN = typename S::LN;
    constexpr int M = S::M, T = S::T, NT = S::NT;
    extern __shared__ __align__(16) float2 sm[];
    float2 *tw = sm, *twr = tw + M, *ex = twr + S::WR, *Zs = ex;
    const int ib = blockIdx.z;
    const int tid = threadIdx.x, p = tid % NPAR, t = (tid / NPAR) % T, row = tid / (NPAR * T);
    const int c = blockIdx.y / a.Nz, z = blockIdx.y - c * a.Nz, y0 = blockIdx.x * 4, y = y0 + row, Nx = a.Nx;
    tw_copy(tw, a.fx.tw, M, tid, NT);
    tw_copy(twr, a.twr, S::WR, tid, NT);
    const bool off = inst_inactive(a, ib);
    pdl_wait();
    pdl_trigger();
    if (off) {
        cpa_wait_all();
        return;
    }
    const float2* in = inst_spec(a, ib) + ((long)c * a.Pz + z) * a.Ny * a.Lx;
    // the thread's columns k and M - k, all loads before the first use
    constexpr int NK = cdiv((M / 8 + 1) * 16, NT);
    float2 Xk[NK], Xm[NK];
#pragma unroll
    for (int i = 0; i < NK; i++) {
        const int e = tid + i * NT, k = (e >> 4) * 4 + (e & 3), r = (e >> 2) & 3;
        const bool in_ = k <= M / 2 && y0 + r < a.Ny;
        Xk[i] = in_ ? in[spec_at(a.Ny, k, y0 + r)] : make_float2(0.f, 0.f);
        Xm[i] = in_ ? in[spec_at(a.Ny, M - k, y0 + r)] : make_float2(0.f, 0.f);
    }
    cpa_wait_all();
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NK; i++) {
        const int e = tid + i * NT, k = (e >> 4) * 4 + (e & 3), r = (e >> 2) & 3;
        if (k > M / 2) continue;
        if (k == 0) { Xk[i].y = 0.f; Xm[i].y = 0.f; }
        const float2 W = twr[k];
        const float2 S1 = make_float2(Xk[i].x + Xm[i].x, Xk[i].y - Xm[i].y);
        const float2 D1 = make_float2(Xk[i].x - Xm[i].x, Xk[i].y + Xm[i].y);
        // T1 = conj(W) D1; Z[k] = S1 + i T1, Z[M-k] = conj(S1) + i conj(T1); both
        // are stored conjugated (the inverse is the conjugate's forward)
        const float2 T1 = make_float2(fma_rn(W.x, D1.x, mul_rn(W.y, D1.y)), fma_rn(W.x, D1.y, -mul_rn(W.y, D1.x)));
        float2* zr = Zs + r * S::ZP;
        zr[k] = make_float2(S1.x - T1.y, -(S1.y + T1.x));
        if (k != 0 && 2 * k != M) zr[M - k] = make_float2(S1.x + T1.y, S1.y - T1.x);
    }
    __syncthreads();
    P2 v[1][LN::NE];
#pragma unroll
    for (int q = 0; q < LN::Qf; q++) {
        const int b = t + T * q;
        if (LN::Bf % T == 0 || b < LN::Bf)
#pragma unroll
            for (int k = 0; k < LN::Rf; k++)
                v[0][q * LN::Rf + k] = p2(Zs[row * S::ZP + NPAR * LN::freq(b, k) + p]);
    }
    __syncthreads();  // the rows become exchange lines
    line_inv<LN, NPAR, 1, 1>(v, t, p, ex + row * S::SR + p * S::SP, 0, tw);
    float* __restrict__ B = inst_B(a, ib, c);
    const int i0 = (z * a.Ny + y) * Nx;
    const bool pairs = (Nx & 1) == 0 && (reinterpret_cast<uintptr_t>(B) & 7) == 0;
    constexpr int H = NPAR == 2 ? (LN::R1 + 1) / 2 : LN::R1;
#pragma unroll
    for (int q = 0; q < LN::Q1; q++)
#pragma unroll
        for (int i = 0; i < H; i++) {
            const int b = t + T * q, j = NPAR == 2 ? i + H * p : i, x = 2 * (b + LN::B1 * j);
            float2 f;
            if constexpr (NPAR == 2) f = f2(line_join<LN, 1, 1>(v, 0, q, i, p));
            else f = f2(v[0][q * LN::R1 + i]);
            if (y < a.Ny && j < LN::R1 && (LN::B1 % T == 0 || b < LN::B1)) {
                if (pairs) {
                    if (x < Nx) *reinterpret_cast<float2*>(B + i0 + x) = make_float2(f.x, -f.y);
                } else {
                    if (x < Nx) B[i0 + x] = f.x;
                    if (x + 1 < Nx) B[i0 + x + 1] = -f.y;
                }
            }
        }
}

// ================================================================ Z
// u[n] W_2H^n for n = N..H-1
template <int H, int N = 1> __device__ __forceinline__ void z_ramp(P2 (&u)[H]) {
    if constexpr (N < H) {
        u[N] = p_twc<N, 2 * H>(u[N]);
        z_ramp<H, N + 1>(u);
    }
}
// One column (kx, y) of one component per thread, planes Ny*Lx apart: the
// frequencies 2r + p of the padded column from the transform of length H of
// x[n] W_2H^(n p).  In place: a thread reads its column before it writes it.
// Streams the spectrum once in and once out: 512x512x32, 114 us forward and
// 125 us inverse for the 605 MB (5.3 and 4.8 TB/s).
template <int H, int NPAR> __global__ void __launch_bounds__(128) k_z_fwd(const __grid_constant__ PassArgs a) {
    const int ib = blockIdx.z;
    const bool off = inst_inactive(a, ib);
    pdl_wait();
    pdl_trigger();
    if (off) return;
    const long ps = (long)a.Ny * a.Lx, e = blockIdx.x * 128L + threadIdx.x;
    if (e >= ps) return;
    float2* col = inst_spec(a, ib) + (long)blockIdx.y * a.Pz * ps + e;
    P2 x[H], u[H];
#pragma unroll
    for (int n = 0; n < H; n++) x[n] = p2(n < a.Nz ? col[n * ps] : make_float2(0.f, 0.f));
#pragma unroll
    for (int n = 0; n < H; n++) u[n] = x[n];
    pdft<H>(u);
#pragma unroll
    for (int k = 0; k < H; k++) col[NPAR * k * ps] = f2(u[k]);
    if constexpr (NPAR == 2) {
        if constexpr (par_dft(H)) {
            pdft_par<H>(x, 1);
        } else {
            z_ramp<H>(x);
            pdft<H>(x);
        }
#pragma unroll
        for (int k = 0; k < H; k++) col[(2 * k + 1) * ps] = f2(x[k]);
    }
}
template <int H, int NPAR> __global__ void __launch_bounds__(128) k_z_inv(const __grid_constant__ PassArgs a) {
    const int ib = blockIdx.z;
    const bool off = inst_inactive(a, ib);
    pdl_wait();
    pdl_trigger();
    if (off) return;
    const long ps = (long)a.Ny * a.Lx, e = blockIdx.x * 128L + threadIdx.x;
    if (e >= ps) return;
    float2* col = inst_spec(a, ib) + (long)blockIdx.y * a.Pz * ps + e;
    P2 u[H], w[H];
    const P2 cj = p2(1.f, -1.f);
#pragma unroll
    for (int k = 0; k < H; k++) u[k] = pmul(p2(col[NPAR * k * ps]), cj);
    if constexpr (NPAR == 2) {
#pragma unroll
        for (int k = 0; k < H; k++) w[k] = pmul(p2(col[(2 * k + 1) * ps]), cj);
        if constexpr (par_dft(H)) {
            pdft_par_t<H>(w, 1);
        } else {
            pdft<H>(w);
            z_ramp<H>(w);
        }
    }
    pdft<H>(u);
#pragma unroll
    for (int n = 0; n < H; n++) {
        if (n < a.Nz) col[n * ps] = f2(pmul(NPAR == 2 ? padd(u[n], w[n]) : u[n], cj));
    }
}

// ================================================================ Y
// lanes: 4 columns fastest, then the parity, then the T threads of a line
template <int L, int NPAR> struct YShape {
    using LN = Line<L>;
    static constexpr int P = NPAR * L, T = LN::T, NT = 4 * NPAR * T, HY = P / 2 + 1;
    static constexpr int LS = pitch16(LN::slots, NPAR == 2 ? 2 : 4);
    static constexpr int lines = 4 * NPAR;
    // exchange buffers: as many of the three components' as leave room for
    // three (L <= 256) or two CTAs per SM beside the kernel block
    static constexpr int NBUF = L <= 192 ? 3 : L <= 384 ? 2 : 1;
    static constexpr size_t smem(int ncomp) {
        return sizeof(float2) * ((size_t)P + (size_t)NBUF * lines * LS) + sizeof(float) * 4 * (size_t)HY * ncomp;
    }
    // registers a thread can have: 6 NE hold the three components' values
    static constexpr int regs = LN::NE <= 8 ? 96 : LN::NE <= 12 ? 128 : NT > 128 ? 128 : 160;
    static constexpr int by_regs = 65536 / (regs * ((NT + 31) / 32 * 32));
    static constexpr int by_smem = (int)(227 * 1024 / (smem(6) + 1024));
    static constexpr int minb0 = by_regs < by_smem ? by_regs : by_smem;
    static constexpr int minb = minb0 < 1 ? 1 : minb0 > 16 ? 16 : minb0;
};

__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// A thread holds the values of all three components (6 NE registers), so that
// the multiply needs no exchange; the kernel block arrives by bulk copies while
// the forward transform runs.  Four columns a CTA: 32-byte pieces times Ny rows
// are one contiguous run.  256x256x16 is bound by issue and shared memory at 12
// warps per SM: 45 us where a 512-point transform in three radix-8 stages took
// 50.5; 512x512x32 by the two exchanges of
// its longer lines (L1 at 67 %, DRAM at a quarter; 1538 us with two columns a CTA,
// whose 16-byte pieces move twice the sectors); small films by one CTA's
// latency (128x128: 4.6 us against 8.3; 250x250: 6.7 against 38.9).
// Kernel components in shared memory: xx yy zz xy (one layer), then yz xz.
template <int L, int NPAR>
__global__ void __launch_bounds__(4 * NPAR * Line<L>::T, YShape<L, NPAR>::minb) k_y(const __grid_constant__ PassArgs a) {
    using S = YShape<L, NPAR>;
    using LN = typename S::LN;
    constexpr int P = S::P, T = S::T, NT = S::NT, HY = S::HY, KS = 4 * HY;
    extern __shared__ __align__(16) float2 sm[];
    float2 *tw = sm, *ex = tw + P;
    float* Ks = reinterpret_cast<float*>(ex + S::NBUF * S::lines * S::LS);  // [comp][ky][4]
    __shared__ __align__(8) uint64_t kbar;
    const int ib = blockIdx.z;
    const int tid = threadIdx.x, w = tid & 3, p = (tid >> 2) & (NPAR - 1), t = tid / (4 * NPAR);
    const int kz = blockIdx.y, kx0 = blockIdx.x * 4, Ny = a.Ny, Pz = a.Pz;
    const int kzm = kz > Pz / 2 ? Pz - kz : kz;
    const float sz = kz > Pz / 2 ? -1.f : 1.f;
    const bool k3d = a.K[3] != nullptr;
    const int ncomp = k3d ? 6 : 4;
    auto karr = [&](int s) { return a.K[s < 3 ? s : s == 3 ? 5 : s - 1]; };
    if (a.Kblocked) {
        if (tid == 0) {
            mbar_init(&kbar, 1);
            mbar_expect_tx(&kbar, (uint32_t)(sizeof(float) * ncomp * KS));
            for (int s = 0; s < ncomp; s++)
                bulk_g2s(Ks + s * KS, karr(s) + kern_idx(a, kzm, 0, kx0, HY), (uint32_t)(sizeof(float) * KS), &kbar);
        }
    } else {  // caller-owned rows
        for (int e = tid; e < ncomp * KS; e += NT) {
            const int s = e / KS, r = e - s * KS, kx = kx0 + (r & 3);
            if (kx < a.Hx) cpa4(Ks + e, karr(s) + kern_idx(a, kzm, r >> 2, kx, HY));
            else Ks[e] = 0.f;
        }
    }
    tw_copy(tw, a.fy.tw, P, tid, NT);
    const bool off = inst_inactive(a, ib);
    pdl_wait();
    pdl_trigger();
    if (off) {  // (not before the copies in flight have landed)
        cpa_wait_all();
        __syncthreads();
        for (int it = 0; a.Kblocked && it < 2 * kTileWaitLimit && !mbar_try_wait(&kbar, 0); it++) {}
        return;
    }
    const long cs = (long)Pz * Ny * a.Lx;
    float2* col = inst_spec(a, ib) + ((long)kz * a.Lx + kx0) * Ny + w;
    P2 v[3][LN::NE];
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
        for (int q = 0; q < LN::Q1; q++)
#pragma unroll
            for (int m = 0; m < LN::R1; m++) {
                const int b = t + T * q, y = b + LN::B1 * m;
                v[c][q * LN::R1 + m] =
                    p2((LN::B1 % T == 0 || b < LN::B1) && y < Ny ? col[c * cs + 4 * y] : make_float2(0.f, 0.f));
            }
    cpa_wait_all();
    __syncthreads();  // twiddles and caller-owned rows are here, barrier initialised
    float2* exl = ex + (w + 4 * p) * S::LS;
    line_fwd<LN, NPAR, 3, S::NBUF>(v, t, p, exl, S::lines * S::LS, tw);
    if (a.Kblocked) {
        for (int it = 0; !mbar_try_wait(&kbar, 0); it++) {
            if (it == kTileWaitLimit && tid == 0) pass_timeout(a, ib);
            if (it >= 2 * kTileWaitLimit) return;
        }
    }
    // kernel multiply (kernmulrsymm3d.cl:41-90), ky mirrored into the stored
    // block; conjugated products: the inverse is conj(FFT(conj(.)))
    auto dot3k = [](P2 x, float kx, P2 y, float ky, P2 z, float kz_) {
        return pfma(z, p2(kz_, -kz_), pfma(y, p2(ky, -ky), pmul(x, p2(kx, -kx))));
    };
#pragma unroll
    for (int q = 0; q < LN::Qf; q++) {
        const int b = t + T * q;
        if (LN::Bf % T == 0 || b < LN::Bf)
#pragma unroll
            for (int k = 0; k < LN::Rf; k++) {
                const int ky = NPAR * LN::freq(b, k) + p, i = q * LN::Rf + k;
                const bool mir = ky > P / 2;
                const float sy = mir ? -1.f : 1.f;
                const float* kr = Ks + (mir ? P - ky : ky) * 4 + w;
                const P2 mx = v[0][i], my = v[1][i], mz = v[2][i];
                const float Kxx = kr[0], Kyy = kr[KS], Kzz = kr[2 * KS], Kxy = kr[3 * KS] * sy;
                if (k3d) {
                    const float Kyz = kr[4 * KS] * (sy * sz), Kxz = kr[5 * KS] * sz;
                    v[0][i] = dot3k(mx, Kxx, my, Kxy, mz, Kxz);
                    v[1][i] = dot3k(mx, Kxy, my, Kyy, mz, Kyz);
                    v[2][i] = dot3k(mx, Kxz, my, Kyz, mz, Kzz);
                } else {
                    v[0][i] = pfma(my, p2(Kxy, -Kxy), pmul(mx, p2(Kxx, -Kxx)));
                    v[1][i] = pfma(my, p2(Kyy, -Kyy), pmul(mx, p2(Kxy, -Kxy)));
                    v[2][i] = pmul(mz, p2(Kzz, -Kzz));
                }
            }
    }
    line_inv<LN, NPAR, 3, S::NBUF>(v, t, p, exl, S::lines * S::LS, tw);
    constexpr int H = NPAR == 2 ? (LN::R1 + 1) / 2 : LN::R1;
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
        for (int q = 0; q < LN::Q1; q++)
#pragma unroll
            for (int i = 0; i < H; i++) {
                const int b = t + T * q, j = NPAR == 2 ? i + H * p : i, y = b + LN::B1 * j;
                float2 f;
                if constexpr (NPAR == 2) f = f2(line_join<LN, 3, 4>(v, c, q, i, p));
                else f = f2(v[c][q * LN::R1 + i]);
                if (j < LN::R1 && (LN::B1 % T == 0 || b < LN::B1) && y < Ny) col[c * cs + 4 * y] = make_float2(f.x, -f.y);
            }
}

}  // namespace umag
