// fft_line.cuh -- mixed-radix line transforms for zero-padded convolutions,
// with two or three register stages and one shared-memory exchange between
// stages.
//
// The convolutions here transform lines of which only the first half carries
// data (open meshes).  The frequencies k = 2r + p of a line of length 2L
// whose upper half is zero are, for each parity p, a transform of length L:
//     X[2r + p] = sum_n (x[n] W_2L^(n p)) W_L^(n r),
// and the first L values of the inverse are the sum over p of two inverse
// transforms of length L.  So a padded line is two dense lines of half the
// length: nothing is loaded, exchanged or multiplied for the padding, and a
// padded length of 512 needs one exchange (256 = 16 x 16) where a 512-point
// transform needs two.  NPAR = 2 for such lines; NPAR = 1 is the plain
// transform of a periodic axis.
//
// L = R1 R2 (R3 = 1) or R1 R2 R3.  Thread t of the T threads of a line owns
// butterflies b = t + T q of every stage.  Forward (decimation in frequency):
//   stage 1: n = b + B1 m,            b < B1 = L/R1, m < R1  -> k1
//   stage 2: b = k1 + R1 n3,          elements n2            -> k2
//   stage 3: b = k1 + R1 k2,          elements n3            -> k3
// with r = k1 + R1 k2 + R1 R2 k3.  k1 runs fastest, so that neighbouring
// threads hold neighbouring frequencies (the kernel rows and half-spectrum rows
// that they touch lie side by side in shared memory) and share the twiddles of n3
// and k2.  With k1 slowest those were 4-way and 2-way bank conflicts in lines of
// three stages: the field of 1024x1024 132 -> 116 us, k_y<512> of 512x512x8 130 -> 123 us (ncu).  The inverse runs the stages backwards on
// the conjugated spectrum with the same (forward) butterflies.  A thread
// writes, between two stages, only the slots that it read before the stage,
// so a buffer needs one barrier per exchange.  The parity factor W_2L^(n p)
// splits into W_2R1^(m p), part of the first butterfly, and W_2L^(b p),
// folded into the twiddles between stages 1 and 2.
//
// All arithmetic is packed FP32 with explicit rounding (fft_packed.cuh): every
// instantiation of a length gives the same bits.
#pragma once
#include "fft_packed.cuh"
#include "fft_pair.cuh"

namespace umag {

// ---------------------------------------------------------------- butterflies
// a - i s d and a + i s d
__device__ __forceinline__ void p_pm_is(P2 a, P2 d, float s, P2& minus_i, P2& plus_i) {
    const P2 ds = pswap(d);
    minus_i = pfma(ds, p2(s, -s), a);
    plus_i = pfma(ds, p2(-s, s), a);
}
__device__ __forceinline__ void pdft3(P2* v) {
    const P2 t = padd(v[1], v[2]), d = psub(v[1], v[2]);
    const P2 m = pfma(t, p2(-0.5f, -0.5f), v[0]);
    v[0] = padd(v[0], t);
    p_pm_is(m, d, 0.86602540378443864676f, v[1], v[2]);
}
__device__ __forceinline__ void pdft5(P2* v) {
    constexpr float c1 = (float)ct_cos(2 * kCtPi / 5), c2 = (float)ct_cos(4 * kCtPi / 5);
    constexpr float s1 = (float)ct_sin(2 * kCtPi / 5), s2 = (float)ct_sin(4 * kCtPi / 5);
    const P2 t1 = padd(v[1], v[4]), t2 = padd(v[2], v[3]), d1 = psub(v[1], v[4]), d2 = psub(v[2], v[3]);
    const P2 m1 = pfma(t2, p2(c2, c2), pfma(t1, p2(c1, c1), v[0]));
    const P2 m2 = pfma(t2, p2(c1, c1), pfma(t1, p2(c2, c2), v[0]));
    const P2 e1 = pfma(d2, p2(s2, s2), pmul(d1, p2(s1, s1)));
    const P2 e2 = pfma(d2, p2(-s1, -s1), pmul(d1, p2(s2, s2)));
    v[0] = padd(v[0], padd(t1, t2));
    p_pm_is(m1, e1, 1.f, v[1], v[4]);
    p_pm_is(m2, e2, 1.f, v[2], v[3]);
}
// u W_L^E for compile-time E
template <int E, int L> __device__ __forceinline__ P2 p_twc(P2 u) {
    constexpr int e = ((E % L) + L) % L;
    if constexpr (e == 0) {
        return u;
    } else if constexpr (4 * e == L) {  // -i
        return pmul(pswap(u), p2(1.f, -1.f));
    } else if constexpr (2 * e == L) {
        return pmul(u, p2(-1.f, -1.f));
    } else if constexpr (4 * e == 3 * L) {  // i
        return pmul(pswap(u), p2(-1.f, 1.f));
    } else {
        constexpr float c = (float)ct_cos(2.0 * kCtPi * e / L), s = -(float)ct_sin(2.0 * kCtPi * e / L);
        return pcmul(u, p2(c, c), p2(-s, s));
    }
}
// y[k1] W_16^(n2 k1) for k1 = K..3
template <int N2, int K = 1> __device__ __forceinline__ void p_tw16(P2* y) {
    if constexpr (K < 4) {
        y[K] = p_twc<N2 * K, 16>(y[K]);
        p_tw16<N2, K + 1>(y);
    }
}
template <int N2 = 0> __device__ __forceinline__ void p_dft16_cols(P2* v, P2 (&y)[4][4]) {
    if constexpr (N2 < 4) {
#pragma unroll
        for (int n1 = 0; n1 < 4; n1++) y[N2][n1] = v[4 * n1 + N2];
        pdft4(y[N2]);
        p_tw16<N2>(y[N2]);
        p_dft16_cols<N2 + 1>(v, y);
    }
}
__device__ __forceinline__ void pdft16(P2* v) {
    P2 y[4][4];  // [n2][k1]
    p_dft16_cols<>(v, y);
#pragma unroll
    for (int k1 = 0; k1 < 4; k1++) {
        P2 z[4] = {y[0][k1], y[1][k1], y[2][k1], y[3][k1]};
        pdft4(z);
#pragma unroll
        for (int k2 = 0; k2 < 4; k2++) v[k1 + 4 * k2] = z[k2];
    }
}
template <int R> __device__ __forceinline__ void pdft(P2* v);
// coprime factors N1 N2 (Good-Thomas: no twiddles): n = N2 n1 + N1 n2,
// k = E1 k1 + E2 k2 (mod N), E1 = 1 (mod N1), 0 (mod N2) and E2 the reverse
template <int N1, int N2, int E1, int E2> __device__ __forceinline__ void pdft_pfa(P2* v) {
    constexpr int N = N1 * N2;
    P2 y[N1][N2];
#pragma unroll
    for (int n1 = 0; n1 < N1; n1++) {
#pragma unroll
        for (int n2 = 0; n2 < N2; n2++) y[n1][n2] = v[(N2 * n1 + N1 * n2) % N];
        pdft<N2>(y[n1]);
    }
#pragma unroll
    for (int k2 = 0; k2 < N2; k2++) {
        P2 z[N1];
#pragma unroll
        for (int n1 = 0; n1 < N1; n1++) z[n1] = y[n1][k2];
        pdft<N1>(z);
#pragma unroll
        for (int k1 = 0; k1 < N1; k1++) v[(E1 * k1 + E2 * k2) % N] = z[k1];
    }
}
// N = 4 N2 (N2 not coprime to 4): y[k1][n2] = DFT4 over n1 of v[N2 n1 + n2],
// times W_N^(n2 k1), DFT_N2 over n2 -> v[k1 + 4 k2]
template <int N2, int J = 0> __device__ __forceinline__ void p_ramp4(P2 (&y)[4][N2]) {
    if constexpr (J < 4 * N2) {
        y[J / N2][J % N2] = p_twc<(J / N2) * (J % N2), 4 * N2>(y[J / N2][J % N2]);
        p_ramp4<N2, J + 1>(y);
    }
}
template <int N2> __device__ __forceinline__ void pdft_4x(P2* v) {
    P2 y[4][N2];
#pragma unroll
    for (int n2 = 0; n2 < N2; n2++) {
        P2 q[4] = {v[n2], v[N2 + n2], v[2 * N2 + n2], v[3 * N2 + n2]};
        pdft4(q);
#pragma unroll
        for (int k1 = 0; k1 < 4; k1++) y[k1][n2] = q[k1];
    }
    p_ramp4<N2>(y);
#pragma unroll
    for (int k1 = 0; k1 < 4; k1++) {
        pdft<N2>(y[k1]);
#pragma unroll
        for (int k2 = 0; k2 < N2; k2++) v[k1 + 4 * k2] = y[k1][k2];
    }
}
// forward DFT of R values, natural order in and out
template <int R> __device__ __forceinline__ void pdft(P2* v) {
    static_assert(R == 1 || R == 2 || R == 3 || R == 4 || R == 5 || R == 6 || R == 8 || R == 10 || R == 12 ||
                      R == 16 || R == 20 || R == 24 || R == 32, "radix");
    if constexpr (R == 2) pdft2(v);
    else if constexpr (R == 3) pdft3(v);
    else if constexpr (R == 4) pdft4(v);
    else if constexpr (R == 5) pdft5(v);
    else if constexpr (R == 6) pdft_pfa<2, 3, 3, 4>(v);
    else if constexpr (R == 8) pdft8(v);
    else if constexpr (R == 10) pdft_pfa<2, 5, 5, 6>(v);
    else if constexpr (R == 12) pdft_pfa<4, 3, 9, 4>(v);
    else if constexpr (R == 16) pdft16(v);
    else if constexpr (R == 20) pdft_pfa<4, 5, 5, 16>(v);
    else if constexpr (R == 24) pdft_pfa<8, 3, 9, 16>(v);
    else if constexpr (R == 32) pdft_4x<8>(v);
}

// ---- DFTs at the frequencies 2k + p of a zero-padded input of 2R values:
// V[k] = sum_m v[m] W_2R^(m (2k + p)), and the transpose
// v[m] = sum_k V[k] W_2R^(m (2k + p)).  For R = 4 N2 the half-bin shift goes
// into the twiddles that the split has anyway (m = N2 n1 + n2, k = k1 + 4 k2:
// W_8^(n1 p), W_2R^(n2 (2 k1 + p))), so it costs no rounding of its own.
// u W_L^(E0 + E1 p)
template <int E0, int E1, int L> __device__ __forceinline__ P2 p_tw_par(P2 u, int p) {
    constexpr float c0 = (float)ct_cos(2.0 * kCtPi * (E0 % L) / L), s0 = -(float)ct_sin(2.0 * kCtPi * (E0 % L) / L);
    constexpr float c1 = (float)ct_cos(2.0 * kCtPi * ((E0 + E1) % L) / L);
    constexpr float s1 = -(float)ct_sin(2.0 * kCtPi * ((E0 + E1) % L) / L);
    const float c = p ? c1 : c0, sn = p ? s1 : s0;
    return pcmul(u, p2(c, c), p2(-sn, sn));
}
constexpr bool par_dft(int R) { return R == 4 || R == 8 || R == 16 || R == 32; }
template <int N2, int J = 0> __device__ __forceinline__ void par_tw(P2 (&y)[4][N2], int p) {
    if constexpr (J < 4 * N2) {  // y[k1][n2] W_(8 N2)^(n2 (2 k1 + p))
        constexpr int k1 = J / N2, n2 = J % N2;
        if constexpr (n2 > 0) y[k1][n2] = p_tw_par<2 * k1 * n2, n2, 8 * N2>(y[k1][n2], p);
        par_tw<N2, J + 1>(y, p);
    }
}
__device__ __forceinline__ void par_w8(P2* q, int p) {  // q[n1] W_8^(n1 p)
    q[1] = p_tw_par<0, 1, 8>(q[1], p);
    q[2] = p_tw_par<0, 2, 8>(q[2], p);
    q[3] = p_tw_par<0, 3, 8>(q[3], p);
}
template <int R> __device__ __forceinline__ void pdft_par(P2* v, int p) {
    constexpr int N2 = R / 4;
    P2 y[4][N2];
#pragma unroll
    for (int n2 = 0; n2 < N2; n2++) {
        P2 q[4] = {v[n2], v[N2 + n2], v[2 * N2 + n2], v[3 * N2 + n2]};
        par_w8(q, p);
        pdft4(q);
#pragma unroll
        for (int k1 = 0; k1 < 4; k1++) y[k1][n2] = q[k1];
    }
    par_tw<N2>(y, p);
#pragma unroll
    for (int k1 = 0; k1 < 4; k1++) {
        pdft<N2>(y[k1]);
#pragma unroll
        for (int k2 = 0; k2 < N2; k2++) v[k1 + 4 * k2] = y[k1][k2];
    }
}
template <int R> __device__ __forceinline__ void pdft_par_t(P2* v, int p) {
    constexpr int N2 = R / 4;
    P2 y[4][N2];
#pragma unroll
    for (int k1 = 0; k1 < 4; k1++) {
#pragma unroll
        for (int k2 = 0; k2 < N2; k2++) y[k1][k2] = v[k1 + 4 * k2];
        pdft<N2>(y[k1]);
    }
    par_tw<N2>(y, p);
#pragma unroll
    for (int n2 = 0; n2 < N2; n2++) {
        P2 q[4] = {y[0][n2], y[1][n2], y[2][n2], y[3][n2]};
        pdft4(q);
        par_w8(q, p);
#pragma unroll
        for (int n1 = 0; n1 < 4; n1++) v[N2 * n1 + n2] = q[n1];
    }
}

// ---------------------------------------------------------------- line shapes
// radices and threads of each line length: stages of at most 16 values, as
// equal as the length allows, a power of two first (pdft_par); T keeps every stage's butterflies on most of
// the threads.  Two-stage lengths exchange once; the longer ones, and those
// without two factors up to 16, twice.
template <int L> struct LineShape;
#define UMAG_LINE(L_, A, B, C, T_) \
    template <> struct LineShape<L_> { static constexpr int R1 = A, R2 = B, R3 = C, T = T_; };
UMAG_LINE(4, 2, 2, 1, 2)
UMAG_LINE(6, 3, 2, 1, 3)
UMAG_LINE(8, 4, 2, 1, 4)
UMAG_LINE(10, 5, 2, 1, 5)
UMAG_LINE(12, 4, 3, 1, 4)
UMAG_LINE(16, 4, 4, 1, 4)
UMAG_LINE(20, 4, 5, 1, 5)
UMAG_LINE(24, 4, 6, 1, 6)
UMAG_LINE(30, 6, 5, 1, 6)
UMAG_LINE(32, 8, 4, 1, 8)
UMAG_LINE(40, 8, 5, 1, 8)
UMAG_LINE(48, 8, 6, 1, 8)
UMAG_LINE(50, 10, 5, 1, 10)
UMAG_LINE(60, 10, 6, 1, 10)
UMAG_LINE(64, 8, 8, 1, 8)
UMAG_LINE(80, 8, 10, 1, 10)
UMAG_LINE(96, 8, 12, 1, 12)
UMAG_LINE(100, 10, 10, 1, 10)
UMAG_LINE(120, 12, 10, 1, 12)
UMAG_LINE(128, 16, 8, 1, 16)
UMAG_LINE(160, 16, 10, 1, 16)
UMAG_LINE(192, 16, 12, 1, 16)
UMAG_LINE(200, 8, 5, 5, 40)
UMAG_LINE(256, 16, 16, 1, 16)
UMAG_LINE(320, 8, 10, 4, 40)
UMAG_LINE(384, 8, 12, 4, 48)
UMAG_LINE(512, 8, 8, 8, 32)
UMAG_LINE(640, 8, 10, 8, 80)
UMAG_LINE(768, 16, 8, 6, 64)
UMAG_LINE(1024, 16, 8, 8, 64)
#undef UMAG_LINE

constexpr int cdiv(int a, int b) { return (a + b - 1) / b; }

template <int L_> struct Line {
    using S = LineShape<L_>;
    static constexpr int L = L_, R1 = S::R1, R2 = S::R2, R3 = S::R3, T = S::T;
    static constexpr bool three = R3 > 1;
    static_assert(R1 * R2 * R3 == L, "radices");
    static constexpr int B1 = L / R1, B2 = L / R2, B3 = three ? L / R3 : 0;
    static constexpr int Q1 = cdiv(B1, T), Q2 = cdiv(B2, T), Q3 = three ? cdiv(B3, T) : 0;
    static constexpr int cmax(int a, int b) { return a > b ? a : b; }
    static constexpr int NE = cmax(Q1 * R1, cmax(Q2 * R2, Q3 * R3));  // values a thread holds
    // exchange slots of (k1, j) (two stages) or (k1, k2 or n2, n3): odd pitches,
    // so that lanes with consecutive butterflies touch different banks
    static constexpr int P2s = R3 | 1, P1s = three ? (R2 * P2s) | 1 : R2 | 1;
    static constexpr int slots = R1 * P1s;
    // values of the thread's final forward stage: Qf butterflies of Rf values
    static constexpr int Rf = three ? R3 : R2, Bf = three ? B3 : B2, Qf = three ? Q3 : Q2;
    // frequency index r of value k of final butterfly b
    __device__ __forceinline__ static int freq(int b, int k) {
        return b + (three ? R1 * R2 : R1) * k;
    }
    static __device__ __forceinline__ int slot1(int k1, int b1) {  // b1 = n2 R3 + n3
        if constexpr (three) return k1 * P1s + (b1 / R3) * P2s + b1 % R3;
        else return k1 * P1s + b1;
    }
    static __device__ __forceinline__ int slot2(int b2, int j) {  // b2 = k1 + R1 n3, j = n2 or k2
        if constexpr (three) return (b2 % R1) * P1s + j * P2s + b2 / R1;
        else return b2 * P1s + j;
    }
    static __device__ __forceinline__ int slot3(int b3, int j) {  // b3 = k1 + R1 k2, j = n3
        return (b3 % R1) * P1s + (b3 / R1) * P2s + j;
    }
};

// Exchange of NC lines held by the same threads, line c through buffer
// c % NBUF (bs slots apart): wr(c) writes the thread's values, rd(c) reads
// them back in the next stage's order.
template <int NC, int NBUF, class W, class R> __device__ __forceinline__ void line_exchange(W wr, R rd) {
#pragma unroll
    for (int c0 = 0; c0 < NC; c0 += NBUF) {
        if (c0 > 0) __syncthreads();  // the buffers' previous lines have been read
#pragma unroll
        for (int c = c0; c < c0 + NBUF && c < NC; c++) wr(c);
        __syncthreads();
#pragma unroll
        for (int c = c0; c < c0 + NBUF && c < NC; c++) rd(c);
    }
}

__device__ __forceinline__ void tw_pair(float2 w, P2& rr, P2& ii) {
    rr = p2(w.x, w.x);
    ii = p2(-w.y, w.y);
}

// the constants W_2R1^(m p) of value m: v *= (p ? W : 1)
template <class LN, int NC, int M = 1> __device__ __forceinline__ void line_parity(P2 (&v)[NC][LN::NE], int q, int p) {
    if constexpr (M < LN::R1) {
        constexpr float cr = (float)ct_cos(kCtPi * M / LN::R1), ci = -(float)ct_sin(kCtPi * M / LN::R1);
        const float wr = p ? cr : 1.f, wi = p ? ci : 0.f;
        const P2 rr = p2(wr, wr), ii = p2(-wi, wi);
#pragma unroll
        for (int c = 0; c < NC; c++) v[c][q * LN::R1 + M] = pcmul(v[c][q * LN::R1 + M], rr, ii);
        line_parity<LN, NC, M + 1>(v, q, p);
    }
}

// butterflies of radix R over the thread's values
template <class LN, int R, int Q, int NC> __device__ __forceinline__ void line_butterflies(P2 (&v)[NC][LN::NE]) {
#pragma unroll
    for (int c = 0; c < NC; c++)
#pragma unroll
        for (int q = 0; q < Q; q++) pdft<R>(&v[c][q * R]);
}

// Forward transform of NC lines.  In: v[c][q R1 + m] = x[b + B1 m]; out:
// v[c][q Rf + k] = X[NPAR freq(b, k) + p], b = t + T q.  ex: the line's slots
// of buffer 0 (buffers bs slots apart); tw: W_(NPAR L)^j for j < NPAR L (shared memory).
template <class LN, int NPAR, int NC, int NBUF>
__device__ __forceinline__ void line_fwd(P2 (&v)[NC][LN::NE], int t, int p, float2* ex, int bs,
                                         const float2* __restrict__ tw) {
    constexpr int R1 = LN::R1, R2 = LN::R2, R3 = LN::R3, T = LN::T;
    if constexpr (NPAR == 2 && par_dft(R1)) {
#pragma unroll
        for (int c = 0; c < NC; c++)
#pragma unroll
            for (int q = 0; q < LN::Q1; q++) pdft_par<R1>(&v[c][q * R1], p);
    } else {
        if constexpr (NPAR == 2) {
#pragma unroll
            for (int q = 0; q < LN::Q1; q++) line_parity<LN, NC>(v, q, p);
        }
        line_butterflies<LN, R1, LN::Q1, NC>(v);
    }
#pragma unroll
    for (int q = 0; q < LN::Q1; q++) {
        const int b = t + T * q;
        if (LN::B1 % T == 0 || b < LN::B1) {
#pragma unroll
            for (int k1 = 0; k1 < R1; k1++) {
                if (NPAR == 1 && k1 == 0) continue;
                P2 rr, ii;
                tw_pair(tw[b * (NPAR * k1 + p)], rr, ii);
#pragma unroll
                for (int c = 0; c < NC; c++) v[c][q * R1 + k1] = pcmul(v[c][q * R1 + k1], rr, ii);
            }
        }
    }
    line_exchange<NC, NBUF>(
        [&](int c) {
            float2* e = ex + (c % NBUF) * bs;
#pragma unroll
            for (int q = 0; q < LN::Q1; q++) {
                const int b = t + T * q;
                if (LN::B1 % T == 0 || b < LN::B1)
#pragma unroll
                    for (int k1 = 0; k1 < R1; k1++) e[LN::slot1(k1, b)] = f2(v[c][q * R1 + k1]);
            }
        },
        [&](int c) {
            const float2* e = ex + (c % NBUF) * bs;
#pragma unroll
            for (int q = 0; q < LN::Q2; q++) {
                const int b = t + T * q;
                if (LN::B2 % T == 0 || b < LN::B2)
#pragma unroll
                    for (int j = 0; j < R2; j++) v[c][q * R2 + j] = p2(e[LN::slot2(b, j)]);
            }
        });
    line_butterflies<LN, R2, LN::Q2, NC>(v);
    if constexpr (LN::three) {
#pragma unroll
        for (int q = 0; q < LN::Q2; q++) {
            const int b = t + T * q;
            if (LN::B2 % T == 0 || b < LN::B2) {
#pragma unroll
                for (int k2 = 1; k2 < R2; k2++) {
                    P2 rr, ii;
                    tw_pair(tw[NPAR * R1 * k2 * (b / R1)], rr, ii);
#pragma unroll
                    for (int c = 0; c < NC; c++) v[c][q * R2 + k2] = pcmul(v[c][q * R2 + k2], rr, ii);
                }
            }
        }
        line_exchange<NC, NBUF>(
            [&](int c) {
                float2* e = ex + (c % NBUF) * bs;
#pragma unroll
                for (int q = 0; q < LN::Q2; q++) {
                    const int b = t + T * q;
                    if (LN::B2 % T == 0 || b < LN::B2)
#pragma unroll
                        for (int j = 0; j < R2; j++) e[LN::slot2(b, j)] = f2(v[c][q * R2 + j]);
                }
            },
            [&](int c) {
                const float2* e = ex + (c % NBUF) * bs;
#pragma unroll
                for (int q = 0; q < LN::Q3; q++) {
                    const int b = t + T * q;
                    if (LN::B3 % T == 0 || b < LN::B3)
#pragma unroll
                        for (int j = 0; j < R3; j++) v[c][q * R3 + j] = p2(e[LN::slot3(b, j)]);
                }
            });
        line_butterflies<LN, R3, LN::Q3, NC>(v);
    }
}

// The reverse: in v[c][q Rf + k] = Y[NPAR freq(b, k) + p] (conjugated by the
// caller), out v[c][q R1 + m] = sum_r Y[NPAR r + p] W^(n (NPAR r + p)), n = b + B1 m:
// this parity's share of the forward transform, which the caller adds up
// over p and conjugates.
template <class LN, int NPAR, int NC, int NBUF>
__device__ __forceinline__ void line_inv(P2 (&v)[NC][LN::NE], int t, int p, float2* ex, int bs,
                                         const float2* __restrict__ tw) {
    constexpr int R1 = LN::R1, R2 = LN::R2, R3 = LN::R3, T = LN::T;
    if constexpr (LN::three) {
        line_butterflies<LN, R3, LN::Q3, NC>(v);  // over k3 -> n3
#pragma unroll
        for (int q = 0; q < LN::Q3; q++) {
            const int b = t + T * q;
            if (LN::B3 % T == 0 || b < LN::B3) {
#pragma unroll
                for (int j = 1; j < R3; j++) {
                    P2 rr, ii;
                    tw_pair(tw[NPAR * R1 * (b / R1) * j], rr, ii);
#pragma unroll
                    for (int c = 0; c < NC; c++) v[c][q * R3 + j] = pcmul(v[c][q * R3 + j], rr, ii);
                }
            }
        }
        line_exchange<NC, NBUF>(
            [&](int c) {
                float2* e = ex + (c % NBUF) * bs;
#pragma unroll
                for (int q = 0; q < LN::Q3; q++) {
                    const int b = t + T * q;
                    if (LN::B3 % T == 0 || b < LN::B3)
#pragma unroll
                        for (int j = 0; j < R3; j++) e[LN::slot3(b, j)] = f2(v[c][q * R3 + j]);
                }
            },
            [&](int c) {
                const float2* e = ex + (c % NBUF) * bs;
#pragma unroll
                for (int q = 0; q < LN::Q2; q++) {
                    const int b = t + T * q;
                    if (LN::B2 % T == 0 || b < LN::B2)
#pragma unroll
                        for (int j = 0; j < R2; j++) v[c][q * R2 + j] = p2(e[LN::slot2(b, j)]);
                }
            });
    }
    line_butterflies<LN, R2, LN::Q2, NC>(v);  // over k2 -> n2
#pragma unroll
    for (int q = 0; q < LN::Q2; q++) {
        const int b = t + T * q;  // k1 + R1 n3
        if (LN::B2 % T == 0 || b < LN::B2) {
            const int kp = NPAR * (b % R1) + p, n3 = b / R1;
#pragma unroll
            for (int j = 0; j < R2; j++) {
                if (!LN::three && j == 0) continue;  // n = 0
                P2 rr, ii;
                tw_pair(tw[(j * R3 + n3) * kp], rr, ii);
#pragma unroll
                for (int c = 0; c < NC; c++) v[c][q * R2 + j] = pcmul(v[c][q * R2 + j], rr, ii);
            }
        }
    }
    line_exchange<NC, NBUF>(
        [&](int c) {
            float2* e = ex + (c % NBUF) * bs;
#pragma unroll
            for (int q = 0; q < LN::Q2; q++) {
                const int b = t + T * q;
                if (LN::B2 % T == 0 || b < LN::B2)
#pragma unroll
                    for (int j = 0; j < R2; j++) e[LN::slot2(b, j)] = f2(v[c][q * R2 + j]);
            }
        },
        [&](int c) {
            const float2* e = ex + (c % NBUF) * bs;
#pragma unroll
            for (int q = 0; q < LN::Q1; q++) {
                const int b = t + T * q;
                if (LN::B1 % T == 0 || b < LN::B1)
#pragma unroll
                    for (int k1 = 0; k1 < R1; k1++) v[c][q * R1 + k1] = p2(e[LN::slot1(k1, b)]);
            }
        });
    if constexpr (NPAR == 2 && par_dft(R1)) {  // over k1 -> m
#pragma unroll
        for (int c = 0; c < NC; c++)
#pragma unroll
            for (int q = 0; q < LN::Q1; q++) pdft_par_t<R1>(&v[c][q * R1], p);
    } else {
        line_butterflies<LN, R1, LN::Q1, NC>(v);
        if constexpr (NPAR == 2) {
#pragma unroll
            for (int q = 0; q < LN::Q1; q++) line_parity<LN, NC>(v, q, p);
        }
    }
}

// Sum over the two parities, held by lanes l and l ^ MASK: the even lane
// keeps the values m < H = ceil(R1/2) of each butterfly, the odd one the
// rest.  Returns the value for slot i < H of butterfly q: m = i + H p.
template <class LN, int NC, int MASK> __device__ __forceinline__ P2 line_join(const P2 (&v)[NC][LN::NE], int c, int q, int i, int p) {
    constexpr int R1 = LN::R1, H = (R1 + 1) / 2;
    const P2 lo = v[c][q * R1 + i], hi = i + H < R1 ? v[c][q * R1 + (i + H < R1 ? i + H : 0)] : lo;
    const P2 keep = p ? hi : lo, give = p ? lo : hi;
    const float2 g = f2(give);
    const float2 r = make_float2(__shfl_xor_sync(0xffffffffu, g.x, MASK), __shfl_xor_sync(0xffffffffu, g.y, MASK));
    return padd(keep, p2(r));
}

}  // namespace umag
