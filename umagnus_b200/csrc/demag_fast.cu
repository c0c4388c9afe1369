// demag_fast.cu -- the fused x/z passes of common three-dimensional sizes, and
// the choice of the pass kernels of a plan.
//
// Pass A: x transform, then z transform of one (y, component) slab in one
// CTA; pass C the reverse.  Compared with separate X and Z passes
// (demag_lines.cuh) the spectrum is written and read once less.
#include <mutex>
#include <set>
#include <utility>

#include "demag_inst.cuh"
#include "fft_pair.cuh"
#include "fft_reg.cuh"
#include "tile.cuh"

namespace umag {

// bulk copies of the passes that gave up waiting (bounded mbarrier poll); the
// plain device-op API reads it after each demag_exec (engine launches report
// the timeout through the controller status instead, PassArgs::fault)
__device__ unsigned g_slab_timeouts = 0;

int demag_timeouts_ptr(unsigned** out) {
    void* p = nullptr;
    UMAG_CUDA(cudaGetSymbolAddress(&p, g_slab_timeouts));
    *out = static_cast<unsigned*>(p);
    return UMAG_OK;
}
int demag_slab_timeouts(unsigned* out, cudaStream_t st) {
    UMAG_CUDA(cudaMemcpyFromSymbolAsync(out, g_slab_timeouts, sizeof(unsigned), 0, cudaMemcpyDeviceToHost, st));
    UMAG_CUDA(cudaStreamSynchronize(st));
    return UMAG_OK;
}
int demag_set_slab_timeouts(unsigned v) {
    UMAG_CUDA(cudaMemcpyToSymbol(g_slab_timeouts, &v, sizeof(unsigned)));
    UMAG_CUDA(cudaDeviceSynchronize());
    return UMAG_OK;
}

constexpr int nz_of_pz(int PZ) { return PZ / 2; }
// offset of spectrum column kx within one (component, kz) plane, y = 0
__device__ __forceinline__ long spec_col(int Ny, int kx) { return spec_at(Ny, kx, 0); }

// ---- passes A and C with the register-blocked FFT (3D, power-of-two sizes)
// x transform: TX = M/8 threads per row (one row per warp or less), rows z
// of one (y, component) slab; z transform: TZ = PZ/8 threads per column.
// Shared memory: staged x and z twiddle tables (RgTw; even slot counts keep
// the later regions 16-byte aligned), the R2C twiddles twr (M), the rows Xs
// [NZ][XP] and the exchange lines (x: one line of LX slots per row, padded
// rg_pad<4> after the first stage and rg_pad<4, 2> after the later ones).
template <int M, int PZ> struct RegAC {
    static constexpr int NZ = nz_of_pz(PZ), TX = M / 8, TZ = PZ / 8, NT = NZ * TX, CPR = NT / TZ;
    static constexpr int XP = ((M + 1 + 11) / 16) * 16 + 4;  // Xs row pitch, = 4 (mod 16) against bank conflicts
    static constexpr int LX = rg_line<M, 4, 2>(), LZ = rg_line<PZ, 3>();
    static constexpr int TWX = (RgTw<M>::size + 1) & ~1, TWZ = (RgTw<PZ>::size + 1) & ~1;
    static constexpr int EXN = NZ * LX > CPR * LZ ? NZ * LX : CPR * LZ;
    static constexpr size_t smem = sizeof(float2) * ((size_t)TWX + TWZ + M + (size_t)NZ * XP + EXN);
    static constexpr bool ok = rg_ok(M) && rg_ok(PZ) && TX <= 32 && PZ % 2 == 0 && NT % TZ == 0 && NT <= 1024;
};

template <int M, int PZ>
__device__ __forceinline__ void k_reg_a_body(const PassArgs& a, const int bx, const int by, const int ib) {
    using S = RegAC<M, PZ>;
    constexpr int NZ = S::NZ, TX = S::TX, TZ = S::TZ, NT = S::NT, CPR = S::CPR, XP = S::XP;
    extern __shared__ __align__(16) float2 sm[];
    float2* twx = sm;             // staged x twiddles (RgTw<M>)
    float2* twz = twx + S::TWX;   // staged z twiddles (RgTw<PZ>)
    float2* twr = twz + S::TWZ;   // M: exp(-2 pi i k / Px)
    float2* Xs = twr + M;         // [NZ][XP]
    float2* ex = Xs + NZ * XP; // exchange lines
    pdl_wait();
    pdl_trigger();
    if (inst_inactive(a, ib)) return;
    const int tid = threadIdx.x;
    const int y = bx, c = by, Ny = a.Ny;
    const float* mp = inst_m(a, ib, c);
    const float msm = inst_msmul(a, ib);
    // x phase: row z, lane t holds packed z[n] = x[2n] + i x[2n+1], n = t + TX*j
    const int z = tid / TX, t = tid % TX;
    float2 v[1][8];
    const int rowi = (z * Ny + y) * M;
    if (a.Ms == nullptr && a.vol == nullptr) {
        // uniform Ms, no geometry: MU0*Ms once, and the pair (x, x+1) in one
        // 8-byte load (scaled_m's rounding: (bsat * 1) * m = bsat * m)
        const float bsat = (float)(kMu0f * (double)msm);
#pragma unroll
        for (int j = 0; j < 8; j++) {
            if (j < 4) {
                const float2 p = *reinterpret_cast<const float2*>(mp + rowi + 2 * (t + TX * j));
                v[0][j] = make_float2(__fmul_rn(bsat, p.x), __fmul_rn(bsat, p.y));
            } else {
                v[0][j] = make_float2(0.f, 0.f);
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < 8; j++) {
            if (j < 4) {  // n < M/2 carries data, the rest is zero padding
                const int i = rowi + 2 * (t + TX * j);
                v[0][j] = make_float2(scaled_m(a, mp, i, msm), scaled_m(a, mp, i + 1, msm));
            } else {
                v[0][j] = make_float2(0.f, 0.f);
            }
        }
    }
    // the twiddle tables while the loads of m are in flight
    for (int i = tid; i < M; i += NT) twr[i] = a.twr[i];
    rg_tw_fill<M>(twx, a.fx.tw, tid, NT);
    if constexpr (PZ != 16 && PZ != 32) rg_tw_fill<PZ>(twz, a.fz.tw, tid, NT);  // (the pair z phase has none)
    __syncthreads();
    rg_fft_fwd<M, 1, true, 4, rg_radix(M, 0) == 8, 2>(v, t, ex + z * S::LX, 0, twx);  // n >= M/2 is zero padding
    // R2C unpack: partner element Z[M-k] lives in lane (TX - t) % TX, element 7-j
    // (or (8-j) & 7 for t = 0); exchanged with warp shuffles.
    const int lane = threadIdx.x & 31;
    const int plane = (lane & ~(TX - 1)) | ((TX - t) & (TX - 1));
    float2 Bv[8];
#pragma unroll
    for (int s = 0; s < 8; s++) {
        float2 r;
        r.x = __shfl_sync(0xffffffffu, v[0][s].x, plane);
        r.y = __shfl_sync(0xffffffffu, v[0][s].y, plane);
        if (t != 0) Bv[7 - s] = r;
        else Bv[(8 - s) & 7] = r;
    }
    float2* xrow = Xs + z * XP;
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const int k = t + TX * j;
        const float2 A = v[0][j], B = Bv[j];
        float2 E = make_float2(0.5f * (A.x + B.x), 0.5f * (A.y - B.y));
        float2 D = make_float2(0.5f * (A.x - B.x), 0.5f * (A.y + B.y));
        float2 O = make_float2(D.y, -D.x);
        float2 W = twr[k];
        float2 WO = make_float2(W.x * O.x - W.y * O.y, W.x * O.y + W.y * O.x);
        xrow[k] = make_float2(E.x + WO.x, E.y + WO.y);
        if (k == 0) xrow[M] = make_float2(A.x - A.y, 0.f);  // Nyquist: Re Z0 - Im Z0
    }
    __syncthreads();
    float2* out = inst_spec(a, ib) + (long)c * PZ * Ny * a.Lx + (long)y * 4;
    const long kzs = (long)Ny * a.Lx;
    if constexpr (PZ == 16 || PZ == 32) {
        // z phase on lane pairs, decimation in frequency: with x[n] = 0 for
        // n >= PZ/2, X[2r + t] = DFT_{PZ/2}( x[n] W_PZ^{n t} )[r], so lane t
        // of a pair produces the kz of parity t from the same PZ/2 inputs --
        // no exchange and no twiddle table.  The DC and Nyquist columns are
        // real in z and share one transform P of (x0 + i xM), split by
        // Hermitian symmetry (X0 = (P[k] + conj P[-k]) / 2, XM = (P[k] -
        // conj P[-k]) / 2i); P[-k] has the parity of k, so it is in the lane.
        constexpr int E2 = PZ / 2, CP2 = NT / 2;
        static_assert(E2 == NZ && M % CP2 == 0, "pair z phase");
        static_assert(NT % 32 == 0, "whole warps of lane pairs");
        // pair partners are lanes l and l ^ 16: a half-warp reads and writes 16
        // consecutive columns of one row
        const int t2 = (tid >> 4) & 1, cl2 = ((tid >> 5) << 4) | (tid & 15);
        const long kM = spec_col(Ny, M);
        // With one column per pair, the (y, component) slab of the blocked
        // spectrum is assembled in the x/z scratch ([kz][kx/4][kx%4], 128-byte
        // aligned; Xs is read into registers first) and written by one bulk
        // tensor store (the slab map pass C loads with), not by 8-byte
        // stores from every thread.
        constexpr bool kSlabShape = M / CP2 == 1;
        const bool slab = kSlabShape && a.slab_map != nullptr && ib == 0 && (smem_u32(Xs) & 15u) == 0;
        const int KB = a.Lx >> 2;
        float2* const sl = Xs + ((128u - (smem_u32(Xs) & 127u)) & 127u) / sizeof(float2);
#pragma unroll
        for (int r0 = 0; r0 < M / CP2; r0++) {
            const int kx = r0 * CP2 + cl2;
            const bool pk = kx == 0;
            float2 u[E2];
#pragma unroll
            for (int n = 0; n < E2; n++) {
                float2 q = Xs[n * XP + kx];
                if (pk) q.y = Xs[n * XP + M].x;
                u[n] = q;
            }
            if (slab) __syncthreads();  // every Xs read is done before the slab overwrites it
            if (t2) tw_ramp<PZ, 1, 0, E2>(u);
            reg_dft<E2>(u);  // u[r] = X[2r + t2]
            if (pk) {
#pragma unroll
                for (int r = 0; r < E2; r++) {
                    const float2 P = u[r], Q = t2 ? u[E2 - 1 - r] : u[(E2 - r) & (E2 - 1)];
                    const int kz = 2 * r + t2;
                    const float2 X0 = make_float2(0.5f * (P.x + Q.x), 0.5f * (P.y - Q.y));
                    const float2 XM = make_float2(0.5f * (P.y + Q.y), -0.5f * (P.x - Q.x));
                    if (slab) {
                        sl[kz * KB * 4] = X0;
                        sl[(kz * KB + (M >> 2)) * 4 + (M & 3)] = XM;
                    } else {
                        out[(long)kz * kzs] = X0;
                        out[(long)kz * kzs + kM] = XM;
                    }
                }
            } else if (slab) {
#pragma unroll
                for (int r = 0; r < E2; r++) sl[((2 * r + t2) * KB + (kx >> 2)) * 4 + (kx & 3)] = u[r];
            } else {
                const long ko = spec_col(Ny, kx);
#pragma unroll
                for (int r = 0; r < E2; r++) out[(long)(2 * r + t2) * kzs + ko] = u[r];
            }
        }
        if (slab) {
            // the block's padding columns M+1 .. 4 KB - 1 (read by no pass) as zeros
            const int padc = 4 * KB - (M + 1);
            for (int e = tid; e < PZ * padc; e += NT) {
                const int kz = e / padc, kx = M + 1 + e % padc;
                sl[(kz * KB + (kx >> 2)) * 4 + (kx & 3)] = make_float2(0.f, 0.f);
            }
            fence_proxy_async();
            __syncthreads();
            if (tid == 0) {
                tma_store_5d(a.slab_map, sl, 0, y, 0, 0, c);
                bulk_commit();
                bulk_wait_read0();
            }
        }
    } else {
        // z phase: column kx, TZ lanes, rows z = tz + TZ*j (zero padding for j >= 4).
        // The DC and Nyquist columns are real in z, so they share one complex
        // transform (x0 + i xM), split afterwards by Hermitian symmetry:
        // X0[k] = (P[k] + conj P[-k]) / 2, XM[k] = (P[k] - conj P[-k]) / 2i.
        // The M - 1 other columns then fill exactly M / CPR = 2 rounds.
        static_assert(M == 2 * CPR, "z rounds: M columns over CPR column groups");
        const int tz = tid % TZ, cl = tid / TZ;
        float2* exz = ex + cl * S::LZ;
    #pragma unroll
        for (int r = 0; r < 2; r++) {
            const int kx = r * CPR + cl;
            const bool pk = kx == 0;
            float2 u[1][8];
    #pragma unroll
            for (int j = 0; j < 8; j++) {
                float2 q = make_float2(0.f, 0.f);
                if (j < 4) {
                    q = Xs[(tz + TZ * j) * XP + kx];
                    if (pk) q.y = Xs[(tz + TZ * j) * XP + M].x;
                }
                u[0][j] = q;
            }
            rg_fft_fwd<PZ, 1, true>(u, tz, exz, 0, twz);
            if (r == 0 && tid < 32) {  // the warp holding column group 0
                const int pl = (lane & ~(TZ - 1)) | ((TZ - tz) & (TZ - 1));
                float2 pr[8];
    #pragma unroll
                for (int s = 0; s < 8; s++) {
                    float2 q;
                    q.x = __shfl_sync(0xffffffffu, u[0][s].x, pl);
                    q.y = __shfl_sync(0xffffffffu, u[0][s].y, pl);
                    if (tz != 0) pr[7 - s] = q;
                    else pr[(8 - s) & 7] = q;
                }
                if (pk) {
    #pragma unroll
                    for (int j = 0; j < 8; j++) {
                        const float2 P = u[0][j], Q = pr[j];
                        out[(tz + TZ * j) * kzs] = make_float2(0.5f * (P.x + Q.x), 0.5f * (P.y - Q.y));
                        out[(tz + TZ * j) * kzs + spec_col(Ny, M)] = make_float2(0.5f * (P.y + Q.y), -0.5f * (P.x - Q.x));
                    }
                    continue;
                }
            }
            const long ko = spec_col(Ny, kx);
    #pragma unroll
            for (int j = 0; j < 8; j++) out[(tz + TZ * j) * kzs + ko] = u[0][j];
        }
    }
}
template <int M, int PZ>
__global__ void __launch_bounds__(RegAC<M, PZ>::NT) k_reg_a(PassArgs a) { k_reg_a_body<M, PZ>(a, blockIdx.x, blockIdx.y, 0); }
// batched: blockIdx.y = index + per * instance (the inst_* views above)
template <int M, int PZ>
__global__ void __launch_bounds__(RegAC<M, PZ>::NT) k_reg_a_bat(PassArgs a) {
    const int per = 3, b = blockIdx.y / per;
    k_reg_a_body<M, PZ>(a, blockIdx.x, blockIdx.y - b * per, b);
}

template <int M, int PZ>
__device__ __forceinline__ void k_reg_c_body(const PassArgs& a, const int bx, const int by, const int ib) {
    using S = RegAC<M, PZ>;
    constexpr int NZ = S::NZ, TX = S::TX, TZ = S::TZ, NT = S::NT, CPR = S::CPR, XP = S::XP;
    extern __shared__ __align__(16) float2 sm[];
    float2* twx = sm;
    float2* twz = twx + S::TWX;
    float2* twr = twz + S::TWZ;
    float2* Xs = twr + M;
    float2* ex = Xs + NZ * XP;
    const bool off = inst_inactive(a, ib);
    pdl_wait();
    pdl_trigger();
    if (off) return;
    const int tid = threadIdx.x;
    // the (y, component) slab of the spectrum by one bulk tensor copy into
    // the x/z scratch (Xs and the exchange lines, idle until the z phase has
    // its inputs in registers): [kz][kx/4][kx%4] complex
    constexpr bool kSlabShape = (PZ == 16 || PZ == 32) && M / (NT / 2) == 1;
    __shared__ __align__(8) uint64_t slab_bar;
    // (Xs is 16-byte aligned, so the 128-byte rounding below moves it by a
    // whole number of float2)
    const bool slab = kSlabShape && a.slab_map != nullptr && ib == 0 && (smem_u32(Xs) & 15u) == 0;
    const int y = bx, c = by, Ny = a.Ny;
    const int KB = a.Lx >> 2;  // four-column blocks per kz row of the slab
    // the copy's destination on a 128-byte boundary (the dynamic region
    // need not start on one; the plan leaves 128 bytes of slack)
    float2* const sl = Xs + ((128u - (smem_u32(Xs) & 127u)) & 127u) / sizeof(float2);
    // the copy is issued first (its initialisation is fenced for the async
    // proxy), so that it is in flight while the twiddle tables are filled;
    // the barrier below makes the initialisation visible to the other threads
    if (slab && tid == 0) {
        mbar_init(&slab_bar, 1);
        mbar_expect_tx(&slab_bar, (uint32_t)(sizeof(float2) * 4 * KB * PZ));
        tma_load_5d(sl, a.slab_map, 0, y, 0, 0, c, &slab_bar);
    }
    for (int i = tid; i < M; i += NT) twr[i] = a.twr[i];
    rg_tw_fill<M>(twx, a.fx.tw, tid, NT);
    if constexpr (PZ != 16 && PZ != 32) rg_tw_fill<PZ>(twz, a.fz.tw, tid, NT);  // (the pair z phase has none)
    __syncthreads();
    if (slab) {
        for (int it = 0; !mbar_try_wait(&slab_bar, 0); it++) {
            if (it == kTileWaitLimit && tid == 0) pass_timeout(a, ib);
            if (it >= 2 * kTileWaitLimit) return;
        }
    }
    const float2* in = inst_spec(a, ib) + (long)c * PZ * Ny * a.Lx + (long)y * 4;
    const long kzs = (long)Ny * a.Lx;
    if constexpr (PZ == 16 || PZ == 32) {
        // z phase on lane pairs, inverse by the conjugate trick, decimation in
        // time: partner t transforms the samples kz = 2j + t (u = conj G),
        // partner 1 scales by W_PZ^k, and the kept outputs z < PZ/2 are
        // X[z] = A[z] + W^z B[z]; partner 0 forms z < PZ/4 and 1 the rest,
        // exchanging one value per output by shuffle.  The DC and Nyquist
        // columns invert to real sequences and share one transform of
        // G0 + i GM (real part -> column 0, imaginary -> column M).
        constexpr int E2 = PZ / 2, H2 = E2 / 2, CP2 = NT / 2;
        static_assert(E2 == NZ && M % CP2 == 0, "pair z phase");
        // pair partners are lanes l and l ^ 16: a half-warp reads and writes 16
        // consecutive columns of one row (conflict-free in shared memory)
        static_assert(NT % 32 == 0, "whole warps of lane pairs");
        const int t2 = (tid >> 4) & 1, cl2 = ((tid >> 5) << 4) | (tid & 15);
        const long kM = spec_col(Ny, M);
#pragma unroll
        for (int r0 = 0; r0 < M / CP2; r0++) {
            const int kx = r0 * CP2 + cl2;
            const bool pk = kx == 0;
            const long ko = spec_col(Ny, kx);
            float2 u[E2];
#pragma unroll
            for (int j = 0; j < E2; j++) {
                const int kz = 2 * j + t2;
                float2 q, g;
                if (slab) {
                    q = sl[(kz * KB + (kx >> 2)) * 4 + (kx & 3)];
                    g = sl[(kz * KB + (M >> 2)) * 4 + (M & 3)];
                } else {
                    q = in[(long)kz * kzs + ko];
                    g = pk ? in[(long)kz * kzs + kM] : make_float2(0.f, 0.f);
                }
                if (pk) q = make_float2(q.x - g.y, q.y + g.x);
                u[j] = make_float2(q.x, -q.y);
            }
            if (slab) __syncthreads();  // every input is in registers before Xs is written
            reg_dft<E2>(u);
            if (t2) tw_ramp<PZ, 1, 0, E2>(u);
#pragma unroll
            for (int i = 0; i < H2; i++) {
                const float2 snd = t2 ? u[i] : u[H2 + i];
                float2 rcv;
                rcv.x = __shfl_xor_sync(0xffffffffu, snd.x, 16);
                rcv.y = __shfl_xor_sync(0xffffffffu, snd.y, 16);
                const float2 own = t2 ? u[H2 + i] : u[i];
                const float2 X = make_float2(own.x + rcv.x, own.y + rcv.y);
                const int z = i + H2 * t2;
                if (pk) {
                    Xs[z * XP] = make_float2(X.x, 0.f);
                    Xs[z * XP + M] = make_float2(-X.y, 0.f);
                } else {
                    Xs[z * XP + kx] = make_float2(X.x, -X.y);
                }
            }
        }
    } else {
        // z phase: inverse transform (conjugate trick) of every column, keep z < NZ.
        // The DC and Nyquist columns invert to real sequences, so they share one
        // transform of G0 + i GM (real part -> column 0, imaginary -> column M);
        // the other columns fill exactly two rounds, whose loads are all issued
        // before the first transform.
        static_assert(M == 2 * CPR, "z rounds: M columns over CPR column groups");
        const int tz = tid % TZ, cl = tid / TZ;
        float2* exz = ex + cl * S::LZ;
        float2 u[2][1][8];
    #pragma unroll
        for (int r = 0; r < 2; r++) {
            const long ko = spec_col(Ny, r * CPR + cl), kM = spec_col(Ny, M);
    #pragma unroll
            for (int j = 0; j < 8; j++) {
                float2 q = in[(tz + TZ * j) * kzs + ko];
                if (r == 0 && cl == 0) {
                    const float2 g = in[(tz + TZ * j) * kzs + kM];
                    q = make_float2(q.x - g.y, q.y + g.x);
                }
                u[r][0][j] = make_float2(q.x, -q.y);
            }
        }
    #pragma unroll
        for (int r = 0; r < 2; r++) {
            const int kx = r * CPR + cl;
            rg_fft_fwd<PZ, 1, true>(u[r], tz, exz, 0, twz);
            if (r == 0 && cl == 0) {
    #pragma unroll
                for (int j = 0; j < 4; j++) {
                    Xs[(tz + TZ * j) * XP] = make_float2(u[r][0][j].x, 0.f);
                    Xs[(tz + TZ * j) * XP + M] = make_float2(-u[r][0][j].y, 0.f);
                }
            } else {
    #pragma unroll
                for (int j = 0; j < 4; j++) Xs[(tz + TZ * j) * XP + kx] = make_float2(u[r][0][j].x, -u[r][0][j].y);
            }
        }
    }
    __syncthreads();
    // x phase: C2R pack Z[k] = (X[k] + conj X[M-k]) + i conj(W^k)(X[k] - conj X[M-k]),
    // inverse transform by the conjugate trick, even/odd samples to B
    const int z = tid / TX, t = tid % TX;
    const float2* xrow = Xs + z * XP;
    float2 v[1][8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const int k = t + TX * j;
        float2 Xk = xrow[k], Xm = xrow[M - k];
        if (k == 0) { Xk.y = 0.f; Xm.y = 0.f; }
        const float2 W = twr[k];
        const float2 S1 = make_float2(Xk.x + Xm.x, Xk.y - Xm.y);
        const float2 D1 = make_float2(Xk.x - Xm.x, Xk.y + Xm.y);
        const float2 T1 = make_float2(W.x * D1.x + W.y * D1.y, W.x * D1.y - W.y * D1.x);
        v[0][j] = make_float2(S1.x - T1.y, -(S1.y + T1.x));  // conj(Z[k])
    }
    rg_fft_fwd<M, 1, true, 4, false, 2>(v, t, ex + z * S::LX, 0, twx);
    float* __restrict__ B = inst_B(a, ib, c);
    const int rowo = (z * Ny + y) * M;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int n = t + TX * j;
        *reinterpret_cast<float2*>(B + rowo + 2 * n) = make_float2(v[0][j].x, -v[0][j].y);
    }
}
// three 512-thread CTAs per SM (40 registers): measured faster for pass C on
// the 256x256x16 multilayer (28.8 -> 27.0 us); pass A keeps two (it spills)
template <int M, int PZ>
__global__ void __launch_bounds__(RegAC<M, PZ>::NT, (RegAC<M, PZ>::NT <= 512 ? 3 : 1))
    k_reg_c(PassArgs a) { k_reg_c_body<M, PZ>(a, blockIdx.x, blockIdx.y, 0); }
// batched: blockIdx.y = index + per * instance (the inst_* views above)
template <int M, int PZ>
__global__ void __launch_bounds__(RegAC<M, PZ>::NT) k_reg_c_bat(PassArgs a) {
    const int per = 3, b = blockIdx.y / per;
    k_reg_c_body<M, PZ>(a, blockIdx.x, blockIdx.y - b * per, b);
}

// ------------------------------------------------------------------ choice of kernels
template <int M, int PZ> static void fill_fused(Passes& f) {
    using S = RegAC<M, PZ>;
    static_assert(S::ok, "register x/z passes");
    f.a = k_reg_a<M, PZ>;
    f.c = k_reg_c<M, PZ>;
    f.ab = k_reg_a_bat<M, PZ>;
    f.cb = k_reg_c_bat<M, PZ>;
    f.smem_ac = S::smem;
    f.ac_scratch = sizeof(float2) * ((size_t)S::NZ * S::XP + S::EXN);
    f.slab_ok = (PZ == 16 || PZ == 32) && M / (S::NT / 2) == 1;
    f.nt_ac = S::NT;
}
// meshes of exactly M x (any) x PZ/2 cells
bool fused_select(int M, int Pz, Passes& f) {
#define AC(m, pz) if (M == m && Pz == pz) { fill_fused<m, pz>(f); return true; }
    AC(64, 16) AC(64, 32) AC(64, 64)
    AC(128, 16) AC(128, 32) AC(128, 64)
    AC(256, 16) AC(256, 32) AC(256, 64)
#undef AC
    return false;
}

bool listed_mesh(const int N[3], const int P[3]) {
    static const int m2[] = {16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512, 1024}, m3[] = {64, 128, 256, 512};
    static const int pz3[] = {12, 16, 32, 64}, py[] = {32, 48, 64, 96, 128, 192, 256, 384, 512, 1024, 2048};
    auto in = [](int v, const int* l, int n) {
        for (int i = 0; i < n; i++)
            if (l[i] == v) return true;
        return false;
    };
    const bool x = P[2] == 1 ? in(N[0], m2, 12) : in(N[0], m3, 4) && in(P[2], pz3, 4);
    return P[0] == 2 * N[0] && x && in(P[1], py, 11);
}

bool lines_select(const int N[3], const int pbc[3], int F[3], Passes& f, bool exact) {
    f = Passes{};
    static const int lens[] = {2, 3, 4, 5, 6, 8, 10, 12, 16, 20, 24, 30, 32, 40, 48, 50, 60, 64, 80, 96, 100, 120, 128,
                               160, 192, 200, 256, 320, 384, 512, 640, 768, 1024};
    auto fits = [&](int need, bool periodic, int unit, auto pick) -> int {
        for (int l : lens) {
            const int have = unit * l;
            if (periodic || exact ? have == need : have >= need)
                if (pick(l)) return have;
        }
        return 0;
    };
    // x: packed pairs of reals, half a padded line of length M per parity
    const int py = pbc[1] ? 1 : 2, pz = pbc[2] ? 1 : 2;
    const int M = pbc[0] ? fits(N[0] / 2, true, 1, [&](int l) { return lines_x(l, 1, f); })
                         : fits(N[0], false, 2, [&](int l) { return lines_x(l, 2, f); });
    const int ly = fits(N[1], pbc[1] != 0, 1, [&](int l) { return lines_y(l, py, f); });
    if (M == 0 || ly == 0) return false;
    F[0] = 2 * M;
    F[1] = py * ly;
    F[2] = 1;
    if (N[2] > 1) {
        const int h = fits(N[2], pbc[2] != 0, 1, [&](int l) { return lines_z(l, pz, f); });
        if (h == 0) return false;
        F[2] = pz * h;
        // the fused passes transform open meshes of exactly their size
        if (!pbc[0] && !pbc[2] && M == N[0] && 2 * N[2] == F[2]) fused_select(M, F[2], f);
    }
    return true;
}

int pass_attrs(void (*k)(PassArgs)) {
    // cudaFuncSetAttribute applies to the current device's context, so the
    // opt-in is made once per device, under a lock (host threads may race):
    // the full 227 KB, and the largest shared-memory carveout, so that several
    // CTAs of these kernels fit on one SM
    static std::mutex mu;
    static std::set<std::pair<int, const void*>> done;
    if (!k) return UMAG_OK;
    int dev = 0;
    UMAG_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    const std::pair<int, const void*> key{dev, reinterpret_cast<const void*>(k)};
    if (done.count(key)) return UMAG_OK;
    cudaFuncAttributes fa;  // the opt-in covers static + dynamic shared memory
    UMAG_CUDA(cudaFuncGetAttributes(&fa, k));
    UMAG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   227 * 1024 - (int)fa.sharedSizeBytes));
    UMAG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    done.insert(key);
    return UMAG_OK;
}

int passes_attrs(const Passes& f) {
    for (auto k : {f.xf, f.xi, f.zf, f.zi, f.y, f.a, f.c, f.ab, f.cb}) UMAG_TRY(pass_attrs(k));
    return UMAG_OK;
}

}  // namespace umag
