// engine.cu -- a whole simulation on the device: effective field, torque,
// RK45DP / RK23 / Heun / RK4 steppers and the step controller.
//
// Restates engine/effectivefield.go, engine/torque.go, engine/rk45dp.go,
// engine/rk23.go, engine/heun.go, engine/rk4.go, engine/stepcontroller.go
// and engine/run.go:150-188 (adaptDt).  The solver state (time, dt in FP64,
// counters, accept/reject decision) lives in device memory and is updated
// by a one-thread controller kernel, so a step never waits for the host and
// many steps are replayed from one CUDA graph.  Buffers are addressed
// through a device-side slot table: accepting a step swaps the state and
// working magnetisation slots and moves k7 into the k1 slot (FSAL,
// engine/stepcontroller.go:76-78) without copying.
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstring>
#include <map>
#include <thread>
#include <vector>

#include "cellmath.cuh"
#include "common.cuh"
#include "demag.cuh"
#include "engine.cuh"
#include "ops.cuh"
#include "tile.cuh"

namespace umag {

// ---------------------------------------------------------------- device state
constexpr double kBoltzmann = 1.380650424e-23;  // mag/constants.go:9 Kb

struct DevCtl {
    float* m;        // state magnetisation (3N, SoA)
    float* mw[2];    // working / stage magnetisations
    float* k[7];     // stage torques
    float* bd;       // demag field of this instance (batched ensembles)
    double t, dt, t0, alarm, stop;
    float h;         // float32(dt * GammaLL) of the step in progress
    int active;      // 0: the step in progress is skipped (stop time reached)
    unsigned int err2, dm2, rel;  // float bit patterns, atomicMax targets
    int nan_seen;
    unsigned arrived;  // CTAs of the step's last torque kernel that are done
    int accepted;
    double last_err, peak_err, last_torque;
    long long nsteps, nundone, nevals;
    int status;
    double max_err, rel_err, min_dt, max_dt, fix_dt, headroom, min_slope, gamma;
    // thermal field: k2 = float32(2 kB / ((GammaLL V) dt)) of the step in
    // progress (engine/temperature.go:111); therm_gv = GammaLL V (0: no thermal field)
    double therm_gv;
    float k2;
};

// Uniform parameters evaluated once on the device with the operations the
// per-cell path uses (bit-identical), so the per-cell kernel does no
// divisions or square roots for them.
struct LocalConsts {
    float inv_ms;  // inv_msat of a uniform Ms (amul.clh:19-26)
    float gilb;    // -1/(1+alpha^2) of a uniform alpha (lltorque2.cl:18)
    float u[3];    // normalised uniform easy axis (uniaxialanisotropy2.cl:19)
    float f1k;     // 2*(K1/Ms) for uniform K1 and Ms
    float f2k;     // 4*(K2/Ms) for uniform K2 and Ms
    PairCoef pc;   // region (0,0) exchange / DMI coefficients
};

// Per-instance uniform parameters of a batched ensemble (one record per
// instance, device memory): the LocalConsts of that instance's material,
// alpha, the applied field and Ms.
struct InstParams {
    LocalConsts kc;
    float alpha_mul, Ms_mul;
    float bext[3];
    int dmi;  // this instance uses the exchange+DMI stencil (engine/exchange.go:49-66: Dind != 0)
};

struct LocalArgs {
    Mesh3 g;
    int N;
    DevCtl* ctl;
    int m_sel;           // 0: ctl->m, 1 and 2: ctl->mw[0] and [1]
    int out_slot;        // torque -> ctl->k[out_slot]
    float* tau_direct;   // if set, torque goes here instead
    float* beff;         // optional B_eff output
    const float* bd;     // demag field or NULL
    const float* aLUT;
    const float* dLUT;
    const uint8_t* regions;
    float wx, wy, wz, cx, cy, cz;
    int dmi, openbc, anis, zeeman, precess;
    const float* frozen;  // FrozenSpins LUT (256) or NULL
    const float* nodemag; // NoDemagSpins LUT (256) or NULL: demag field zeroed there
    int cubic;            // cubic anisotropy on (cp)
    CubicParams cp;
    const float* dbLUT;   // bulk DMI LUT or NULL
    int thermal;          // thermal field on (off while relaxing)
    const float* temp;
    float temp_mul;
    unsigned long long seed;
    int ms_uniform, alpha_uniform, anis_uniform;
    DmiPairLut dl;
    LocalConsts kc;
    UniaxParams up;
    const float* bext[3];
    const float* alpha;
    float alpha_mul;
    const float* Ms;
    float Ms_mul;
    const InstParams* ip;  // batched: per-instance parameters (uniform maps only)
    int early;             // demag passes precede the kernel: only its demag field has to be waited for
    const float* mbuf[2];  // the second and third magnetisation buffers (select the tile map)
};

__global__ void k_local_consts(LocalArgs a, LocalConsts* out) {
    LocalConsts c{};
    c.inv_ms = a.Ms_mul == 0.0f ? 0.0f : fd(1.0f, a.Ms_mul);
    c.gilb = fd(-1.0f, fa(1.0f, fm(a.alpha_mul, a.alpha_mul)));
    f3 u{a.up.ux_mul, a.up.uy_mul, a.up.uz_mul};
    float len = __fsqrt_rn(dot3(u, u));
    float il = (len != 0.0f) ? fd(1.0f, len) : 0.0f;
    c.u[0] = fm(il, u.x); c.u[1] = fm(il, u.y); c.u[2] = fm(il, u.z);
    c.f1k = fm(2.0f, fm(a.up.K1_mul, c.inv_ms));
    c.f2k = fm(4.0f, fm(a.up.K2_mul, c.inv_ms));
    const float A = a.aLUT[0];
    c.pc.wax = fm(a.wx, A);
    c.pc.way = fm(a.wy, A);
    c.pc.waz = fm(a.wz, A);
    const float D = a.dLUT ? a.dLUT[0] : 0.0f;
    c.pc.sx = fd(fm(2.0f, A), fm(a.cx, a.cx));
    c.pc.sy = fd(fm(2.0f, A), fm(a.cy, a.cy));
    c.pc.sz = fd(fm(2.0f, A), fm(a.cz, a.cz));
    c.pc.dcx = fd(D, a.cx);
    c.pc.dcy = fd(D, a.cy);
    const float t = fd(fm(0.5f, D), A);
    c.pc.qx = fm(a.cx, t);
    c.pc.qy = fm(a.cy, t);
    *out = c;
}

// DMI coefficients per region pair (see DmiPairLut)
__global__ void k_dmi_pairs(const float* __restrict__ aLUT, const float* __restrict__ dLUT, float cx, float cy,
                            float cz, float* sx, float* sy, float* sz, float* dcx, float* dcy, float* qx, float* qy,
                            int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float A = aLUT[i], D = dLUT[i];
        sx[i] = fd(fm(2.0f, A), fm(cx, cx));
        sy[i] = fd(fm(2.0f, A), fm(cy, cy));
        sz[i] = fd(fm(2.0f, A), fm(cz, cz));
        dcx[i] = fd(D, cx);
        dcy[i] = fd(D, cy);
        float t = fd(fm(0.5f, D), A);
        qx[i] = fm(cx, t);
        qy[i] = fm(cy, t);
    }
}

// ---------------------------------------------------------------- controller
__device__ void adapt_dt(DevCtl* c, double corr) {
    if (c->fix_dt != 0) { c->dt = c->fix_dt; return; }
    if (isnan(corr)) corr = 1;
    if (corr == 0) { c->status = 1; return; }
    corr *= c->headroom;
    if (corr > 2) corr = 2;
    if (corr < 1. / 2.) corr = 1. / 2.;
    c->dt *= corr;
    if (c->min_dt != 0 && c->dt < c->min_dt) c->dt = c->min_dt;
    if (c->max_dt != 0 && c->dt > c->max_dt) c->dt = c->max_dt;
    // the float32 step h = dt*GammaLL, times the largest tableau coefficient
    // (|-355/33| < 16), must stay finite: zero torque (err = 0) doubles dt
    // every step, and an infinite h turns the stages into Inf*0 = NaN
    if (c->dt * c->gamma > 0x1p120) c->dt = 0x1p120 / c->gamma;
    if (c->dt == 0) { c->status = 2; return; }
    if (c->t < c->alarm && c->t + c->dt > c->alarm) c->dt = c->alarm - c->t;
    if (!(c->dt > 0)) c->status = 3;
}

// engine/rk45dp.go:16-50 (start of Step): fixed dt, h, t0, clear maxima;
// skip the step once the run's stop time is reached (engine/run.go:212-231).
// Every CTA of a first stage kernel evaluates step_runs and step_h; one of
// its threads also runs step_begin, which changes nothing that they read.
__device__ __forceinline__ bool step_runs(const DevCtl* c) { return c->t < c->stop && c->status == 0; }
__device__ __forceinline__ float step_h(const DevCtl* c) {
    return (float)((c->fix_dt != 0 ? c->fix_dt : c->dt) * c->gamma);
}
__device__ __forceinline__ void step_begin(DevCtl* c) {
    c->active = step_runs(c);
    if (!c->active) return;
    if (c->fix_dt != 0) c->dt = c->fix_dt;
    c->h = (float)(c->dt * c->gamma);
    if (c->therm_gv != 0) c->k2 = (float)(2 * kBoltzmann / (c->therm_gv * c->dt));
    c->t0 = c->t;
    c->err2 = 0u; c->dm2 = 0u; c->rel = 0u;
    c->arrived = 0u;
    c->accepted = 0;
}
__global__ void k_step_begin(DevCtl* c0, int nb) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;  // one thread per instance
    pdl_wait();
    pdl_trigger();
    if (b < nb) step_begin(c0 + b);
}

// what the controller of a stepper does after its last evaluation
struct CtlArgs {
    int kind, acc, rej;      // controller and its exponents, below
    int fsal_from, fsal_to;  // k slots swapped on acceptance (-1: none)
    int nevals;
    int new_m;               // the working buffer (1, 2) that becomes the state
    int rk4;                 // record max |k4| (setMaxTorque, engine/rk4.go:64)
};

// kind 0: integralController (engine/stepcontroller.go:35-97), FSAL when fsal
// kind 1: simpleController (:13-32, RK4); kind 2: Heun (engine/heun.go:40-58)
// kind 3: Euler (engine/euler.go:16-35), always accepted
__device__ void controller(DevCtl* c, const CtlArgs& q) {
    const int kind = q.kind, acc = q.acc, rej = q.rej;
    c->nevals += q.nevals;
    if (c->nan_seen) c->status = 4;
    if (kind == 3) {
        // setMaxTorque(dy0), then dt = FixDt, or float32(MaxErr / LastTorque)
        // treated as the largest allowed change of m; h is the float32 dt*GammaLL
        const double lt = sqrt((double)__uint_as_float(c->dm2));
        c->last_torque = lt;
        float hf;
        if (c->fix_dt != 0) {
            c->dt = c->fix_dt;
            hf = (float)(c->dt * c->gamma);
        } else {
            hf = (float)(c->max_err / lt);
            c->dt = (double)hf / c->gamma;
        }
        if (!(hf > 0.0f)) {  // euler.go:32 "Euler solver requires fixed time step > 0"
            c->status = 5;
            c->accepted = 0;
            return;
        }
        c->h = hf;
        const double err = (double)hf * lt;
        c->last_err = err;
        if (err > c->peak_err) c->peak_err = err;
        c->t = c->t0 + c->dt;
        c->nsteps++;
        c->accepted = 1;
        return;
    }
    double h = (double)c->h;
    double err = sqrt((double)__uint_as_float(c->err2)) * h;
    double maxdm = sqrt((double)__uint_as_float(c->dm2));
    bool ok = err < c->max_err || c->dt <= c->min_dt || c->fix_dt != 0;
    if (kind == 0) {
        if (ok) {
            int fail = 0;
            double rlerr = 0.0;
            if (!(maxdm < c->min_slope)) {
                rlerr = (double)__uint_as_float(c->rel);
                fail = 1;
            }
            if (fail == 0 || c->rel_err <= 0.0 || rlerr < c->rel_err || c->dt <= c->min_dt || c->fix_dt != 0) {
                c->last_err = err;
                if (err > c->peak_err) c->peak_err = err;
                c->last_torque = maxdm;
                c->nsteps++;
                c->t = c->t0 + c->dt;
                adapt_dt(c, fail == 0 ? pow(c->max_err / err, 1. / acc) : pow(c->rel_err / rlerr, 1. / acc));
                c->accepted = 1;
            } else {
                c->t = c->t0;
                c->nundone++;
                adapt_dt(c, pow(c->rel_err / rlerr, 1. / rej));
            }
        } else {
            c->t = c->t0;
            c->nundone++;
            adapt_dt(c, pow(c->max_err / err, 1. / rej));
        }
    } else if (kind == 1) {  // RK4: Time = t0 + dt was set before stage 4 (rk4.go:51)
        c->t = c->t0 + c->dt;
        if (ok) {
            c->nsteps++;
            adapt_dt(c, pow(c->max_err / err, 1. / acc));
            c->last_err = err;
            if (err > c->peak_err) c->peak_err = err;
            c->accepted = 1;
        } else {
            c->nundone++;
            adapt_dt(c, pow(c->max_err / err, 1. / rej));
            c->t = c->t0;
        }
    } else {  // Heun: time was advanced before the second evaluation
        if (ok) {
            c->t = c->t0 + c->dt;
            c->nsteps++;
            adapt_dt(c, pow(c->max_err / err, 1. / 2.));
            c->last_err = err;
            if (err > c->peak_err) c->peak_err = err;
            c->last_torque = maxdm;
            c->accepted = 1;
        } else {
            c->t = c->t0;
            c->nundone++;
            adapt_dt(c, pow(c->max_err / err, 1. / 3.));
        }
    }
    if (c->accepted && kind == 0 && q.fsal_from >= 0) {
        float* t = c->k[q.fsal_to];
        c->k[q.fsal_to] = c->k[q.fsal_from];
        c->k[q.fsal_from] = t;
    }
}

// Controller and end of the step, by one thread once every CTA of the step's
// last evaluation has added its maxima.  Accepted: the working
// magnetisation becomes the state (pointer swap); the steppers that form
// their solution afterwards (Euler, Heun, RK4) write it to the new state
// buffer from the old one.
__device__ __noinline__ void step_finish(DevCtl* c, const CtlArgs& q) {
    // other CTAs' atomics: read past this SM's L1
    c->err2 = __ldcg(&c->err2);
    c->dm2 = __ldcg(&c->dm2);
    c->rel = __ldcg(&c->rel);
    c->nan_seen = __ldcg(&c->nan_seen);
    controller(c, q);
    if (c->accepted) {
        float* t = c->m;
        c->m = c->mw[q.new_m - 1];
        c->mw[q.new_m - 1] = t;
        if (q.rk4) c->last_torque = sqrt((double)__uint_as_float(c->dm2));
    }
}

// ---------------------------------------------------------------- after an evaluation
constexpr int kMaxTerms = 7;
// What the torque kernel does with a cell's torque besides storing it (or, where
// fuse_tails says so, kernels of their own).
// kStage: the next working magnetisation, dst = normalize(m + sum_j (c_j h)
// k_j) with Madd<n> rounding (opencl/madd.go, madd<n>.cl) then normalize2.cl;
// the cell's own torque is the last term.  kErr: the error estimate
// sum_j e_j k_j and its maxima, again with the torque as the last term; the
// last CTA to finish runs the controller.
enum { kNoTail = 0, kStageTail = 1, kErrTail = 2 };
struct TailArgs {
    int kind = kNoTail;
    int nk = 0;              // stored torques that take part
    int slot[kMaxTerms];
    float c[kMaxTerms];      // float32 constants of those and (at nk) of the cell's own torque
    int dst = 0;             // stage: 1 or 2, ctl->mw
    int normalize = 0;
    const float* vol = nullptr;
    int heun = 0;            // error = |k - own| (MaxVecDiff)
    CtlArgs ctl{};
};
__device__ __forceinline__ float* mbuf(const DevCtl* c, int sel) { return sel == 0 ? c->m : c->mw[sel - 1]; }

// Values a cell's tail needs from memory; requested before the stencil, so
// that they arrive while the field is summed.
struct TailIn {
    f3 m, k[5];
    float vol;
};
template <int TAIL> __device__ __forceinline__ void tail_load(TailIn& in, const TailArgs& ta, const DevCtl* ctl, int N, int I) {
    if constexpr (TAIL != kNoTail) {
#pragma unroll
        for (int j = 0; j < 5; j++)
            if (j < ta.nk) {
                const float* k = ctl->k[ta.slot[j]];
                in.k[j] = f3{k[I], k[N + I], k[2 * N + I]};
            }
    }
    if constexpr (TAIL == kStageTail) {
        in.m = f3{ctl->m[I], ctl->m[N + I], ctl->m[2 * N + I]};
        in.vol = ta.vol ? __ldg(ta.vol + I) : 1.0f;
    }
}
// one component of the stage (x: values of the terms nk.., factors fac)
__device__ __forceinline__ float stage_comb(int nk, const float (&fac)[6], float m, const float (&k)[5], float t) {
    if (nk == 1) return fa(fm(1.0f, m), fa(fm(fac[0], k[0]), fm(fac[1], t)));  // madd3
    float acc = fm(1.0f, m);
    float ft = fac[0];
#pragma unroll
    for (int j = 0; j < 5; j++)
        if (j < nk) {
            acc = fa(acc, fm(fac[j], k[j]));
            ft = fac[j + 1];
        }
    return fa(acc, fm(ft, t));
}
__device__ __forceinline__ void stage_tail(const TailIn& in, const TailArgs& ta, const DevCtl* ctl, int N, int I, f3 t) {
    const float h = ctl->h;
    float fac[6];
#pragma unroll
    for (int j = 0; j < 6; j++) fac[j] = fm(ta.c[j], h);
    const float kx[5] = {in.k[0].x, in.k[1].x, in.k[2].x, in.k[3].x, in.k[4].x};
    const float ky[5] = {in.k[0].y, in.k[1].y, in.k[2].y, in.k[3].y, in.k[4].y};
    const float kz[5] = {in.k[0].z, in.k[1].z, in.k[2].z, in.k[3].z, in.k[4].z};
    f3 v{stage_comb(ta.nk, fac, in.m.x, kx, t.x), stage_comb(ta.nk, fac, in.m.y, ky, t.y),
         stage_comb(ta.nk, fac, in.m.z, kz, t.z)};
    if (ta.normalize) v = normalize_vol(v, in.vol);
    float* d = mbuf(ctl, ta.dst);
    d[I] = v.x; d[N + I] = v.y; d[2 * N + I] = v.z;
}
// max |Err|^2, max |delM|^2 and max |Err|/|delM| of one cell (VecNorm + Div +
// MaxAbs of stepcontroller.go:51-63); Err itself is never written to memory.
// NaNs are ignored like the reference's fmax and reported apart.
struct ErrMax {
    float e2 = 0.f, d2 = 0.f, rel = 0.f;
    int nan = 0;
};
__device__ __forceinline__ ErrMax err_tail(const TailIn& in, const TailArgs& ta, f3 t) {
    auto comb = [&](const float (&k)[5], float x) {
        if (ta.heun) return fs(ta.nk ? k[0] : x, x);
        float acc = fm(ta.c[0], k[0]), ct = ta.c[1];
#pragma unroll
        for (int j = 1; j < 5; j++)
            if (j < ta.nk) {
                acc = fa(acc, fm(ta.c[j], k[j]));
                ct = ta.c[j + 1];
            }
        return fa(acc, fm(ct, x));
    };
    const float kx[5] = {in.k[0].x, in.k[1].x, in.k[2].x, in.k[3].x, in.k[4].x};
    const float ky[5] = {in.k[0].y, in.k[1].y, in.k[2].y, in.k[3].y, in.k[4].y};
    const float kz[5] = {in.k[0].z, in.k[1].z, in.k[2].z, in.k[3].z, in.k[4].z};
    const f3 E{comb(kx, t.x), comb(ky, t.y), comb(kz, t.z)};
    const float e2 = dot3(E, E), d2 = dot3(t, t);
    const float en = __fsqrt_rn(e2), dn = __fsqrt_rn(d2);
    const float r = dn == 0.0f ? 0.0f : fd(en, dn);
    return ErrMax{fmaxf(0.f, e2), fmaxf(0.f, d2), fmaxf(0.f, r), (e2 != e2) | (d2 != d2)};
}
// The CTA's maxima to the controller record; the last of the instance's ncta
// CTAs then runs the controller.  Whole warps (block sizes are multiples of 32).
// The record is read before it is updated: maxima settle after a few CTAs, and
// tens of thousands of atomics on one address would bound a large mesh.
__device__ __forceinline__ void err_finish(const ErrMax& v, bool ok, const TailArgs& ta, DevCtl* ctl, unsigned ncta) {
    __shared__ unsigned sh[4][8];
    const int tid = threadIdx.y * blockDim.x + threadIdx.x, nw = (blockDim.x * blockDim.y) >> 5;
    const unsigned e = __reduce_max_sync(0xffffffffu, __float_as_uint(v.e2));
    const unsigned d = __reduce_max_sync(0xffffffffu, __float_as_uint(v.d2));
    const unsigned r = __reduce_max_sync(0xffffffffu, __float_as_uint(v.rel));
    const unsigned n = __reduce_or_sync(0xffffffffu, (unsigned)v.nan | (ok ? 0u : 2u));
    if ((tid & 31) == 0) {
        sh[0][tid >> 5] = e; sh[1][tid >> 5] = d; sh[2][tid >> 5] = r; sh[3][tid >> 5] = n;
    }
    __syncthreads();  // (and every read of the record by this CTA is done)
    if (tid != 0) return;
    unsigned me = 0, md = 0, mr = 0, mn = 0;
    for (int w = 0; w < nw; w++) {
        me = max(me, sh[0][w]); md = max(md, sh[1][w]); mr = max(mr, sh[2][w]); mn |= sh[3][w];
    }
    if (me > __ldcg(&ctl->err2)) atomicMax(&ctl->err2, me);
    if (md > __ldcg(&ctl->dm2)) atomicMax(&ctl->dm2, md);
    if (mr > __ldcg(&ctl->rel)) atomicMax(&ctl->rel, mr);
    if (mn & 1) atomicOr(&ctl->nan_seen, 1);
    if (mn & 2) return;  // a wait gave up: the status says so, and the step does not end
    __threadfence();
    if (atomicAdd(&ctl->arrived, 1u) + 1u == ncta) {
        __threadfence();
        step_finish(ctl, ta.ctl);
    }
}

__device__ __forceinline__ f3 lltorque_g(f3 m, f3 H, float alpha, float gilb) {
    f3 mxH = cross3(m, H);
    f3 mmxH = cross3(m, mxH);
    return f3{fm(gilb, fa(mxH.x, fm(alpha, mmxH.x))), fm(gilb, fa(mxH.y, fm(alpha, mmxH.y))),
              fm(gilb, fa(mxH.z, fm(alpha, mmxH.z)))};
}

// engine/effectivefield.go:14-24 + engine/torque.go:135-144 for one cell:
// B = demag; B += exchange(+DMI)/Ms; B += anisotropy; B += B_ext; torque.
// UREG: every cell is in region 0 (no region map), so the region-pair
// coefficients are scalars and no region is loaded.  TILE (with UREG, not
// BAT, non-periodic mesh): the CTA's magnetisation tile with its halo comes
// into shared memory by one TMA load (tile.cuh) and the stencils read it.
// UNI (with UREG, not BAT): a uniform material with only the common terms --
// uniform Ms, alpha and anisotropy, precession on, no OpenBC, and no
// NoDemagSpins, bulk DMI, cubic anisotropy, thermal field, FreezeSpins or
// B_eff output --
// so that those tests and branches leave the instruction stream; the
// arithmetic is the same operations in the same order.
template <bool UREG, bool BAT, bool TILE, bool UNI, int TAIL>
__global__ void __launch_bounds__(256) k_local_torque(const __grid_constant__ LocalArgs a,
                                                      const __grid_constant__ TileMaps tm,
                                                      const __grid_constant__ TailArgs ta) {
    static_assert(!TILE || (UREG && !BAT), "tiles: region-free, not batched");
    static_assert(!UNI || (UREG && !BAT), "uniform material: region-free, not batched");
    // BAT: blockIdx.z = iz + Nz * instance; the instance's controller,
    // demag field and uniform parameters replace the shared ones
    static_assert(!BAT || UREG, "batched ensembles have no region maps");
    // behind the demag passes everything but the demag field was written by
    // kernels before the last one: it is loaded, and the stencil summed, while
    // the last pass runs (common.cuh)
    if (!a.early) {
        pdl_wait();
        pdl_trigger();
    }
    int iz = blockIdx.z;
    DevCtl* ctl = a.ctl;
    const float* bd = a.bd;
    const LocalConsts* kcp = &a.kc;
    float alpha_mul = a.alpha_mul;
    const InstParams* ip = nullptr;
    if constexpr (BAT) {
        const int b = iz / a.g.Nz;
        iz -= b * a.g.Nz;
        ctl += b;
        bd = ctl->bd;
        ip = a.ip + b;
        kcp = &ip->kc;
        alpha_mul = ip->alpha_mul;
    }
    const LocalConsts& kc = *kcp;
    const bool dmi = BAT ? ip->dmi != 0 : a.dmi != 0;
    if (!ctl->active) {
        pdl_wait();
        return;
    }
    int ix = blockIdx.x * blockDim.x + threadIdx.x;
    int iy = blockIdx.y * blockDim.y + threadIdx.y;
    const int N = a.N;
    const float* m = mbuf(ctl, a.m_sel);
    const float *mx = m, *my = m + N, *mz = m + 2 * N;
    TileView tv{};
    bool live = true;  // the tile arrived
    if constexpr (TILE) {
        extern __shared__ __align__(128) float tile_raw[];
        __shared__ __align__(8) uint64_t bar;
        // the copy's destination on a 128-byte boundary whatever the offset of
        // the dynamic region (launched with 128 bytes of slack)
        float* const tile = tile_raw + ((128u - (smem_u32(tile_raw) & 127u)) & 127u) / sizeof(float);
        const bool three_d = a.g.Nz > 1;
        const uint32_t bytes = (uint32_t)tile_bytes(blockDim.x, blockDim.y, a.g.Nz);
        const bool leader = threadIdx.x == 0 && threadIdx.y == 0;
        if (leader) mbar_init(&bar, 1);
        __syncthreads();
        if (leader) {
            mbar_expect_tx(&bar, bytes);
            tma_load_4d(tile, &tm.map[m == a.mbuf[0] ? 1 : m == a.mbuf[1] ? 2 : 0], (int)(blockIdx.x * blockDim.x) - kTileHaloX,
                        (int)(blockIdx.y * blockDim.y) - 1, three_d ? iz - 1 : iz, 0, &bar);
        }
        // bounded wait: past the limit flag the failure, wait once more for
        // the copy in flight, and leave without writing
        for (int it = 0; live && !mbar_try_wait(&bar, 0); it++) {
            if (it == kTileWaitLimit && leader) atomicCAS(&ctl->status, 0, 7);
            if (it >= 2 * kTileWaitLimit) live = false;
        }
        tv = TileView{tile, tile_pitch(blockDim.x), tile_rows(blockDim.y), three_d ? 3 : 1, three_d ? 1 : 0};
    }
    const bool cell = live && ix < a.g.Nx && iy < a.g.Ny;
    if (!cell && a.early) pdl_wait();
    if (TAIL != kErrTail && !cell) return;
    ErrMax err{};
    if (cell) {
        int I = (iz * a.g.Ny + iy) * a.g.Nx + ix;
        TailIn in{};
        tail_load<TAIL>(in, ta, ctl, N, I);
        f3 m0;
        if constexpr (TILE) m0 = tv.at(threadIdx.x, threadIdx.y, 0, 0, 0);
        else m0 = ld3(mx, my, mz, I);
        const bool magnetic = !is0(m0);
        f3 e{0.f, 0.f, 0.f};
        float inv = 0.f;
        if (magnetic) {
            if constexpr (TILE) {
                e = dmi ? dmi_sum_tile<UNI>(tv, threadIdx.x, threadIdx.y, kc.pc, a.openbc != 0, a.g.Nz > 1, m0)
                        : exchange_sum_tile(tv, threadIdx.x, threadIdx.y, kc.pc, a.g.Nz > 1, m0);
            } else if (!BAT && !UNI && a.dbLUT) {  // engine/exchange.go:60-61 AddDMIBulk
                e = dmibulk_sum(mx, my, mz, a.aLUT, a.dbLUT, a.regions, a.cx, a.cy, a.cz, a.g, a.openbc != 0, ix, iy,
                                iz, m0, UREG ? 0 : __ldg(a.regions + I));
            } else if constexpr (UREG) {
                e = dmi ? dmi_sum_u(mx, my, mz, kc.pc, a.g, a.openbc != 0, ix, iy, iz, m0)
                        : exchange_sum_u(mx, my, mz, kc.pc, a.g, ix, iy, iz, m0);
            } else {
                int r0 = __ldg(a.regions + I);
                e = a.dmi ? dmi_sum_lut(mx, my, mz, a.dl, a.regions, a.g, a.openbc != 0, ix, iy, iz, m0, r0)
                          : exchange_sum(mx, my, mz, a.aLUT, a.regions, a.wx, a.wy, a.wz, a.g, ix, iy, iz, m0, r0);
            }
            inv = (BAT || UNI || a.ms_uniform) ? kc.inv_ms : inv_msat(a.Ms, a.Ms_mul, I);
        }
        if (a.early) {
            pdl_wait();
            pdl_trigger();
        }
        f3 B{0.f, 0.f, 0.f};
        if (bd) B = f3{bd[I], bd[N + I], bd[2 * N + I]};
        // engine/demag.go:95-97: NoDemagSpins cells feel no demag field
        if (!BAT && !UNI && a.nodemag && __ldg(a.nodemag + (UREG ? 0 : __ldg(a.regions + I))) != 0.0f) B = f3{0.f, 0.f, 0.f};
        if (magnetic) {
            B.x = fa(B.x, fm(e.x, inv));
            B.y = fa(B.y, fm(e.y, inv));
            B.z = fa(B.z, fm(e.z, inv));
        }
        if (a.anis) {
            if (BAT || UNI || a.anis_uniform) {  // uniaxialanisotropy2.cl:27-34 with the uniform factors hoisted
                f3 u{kc.u[0], kc.u[1], kc.u[2]};
                float mu = dot3(m0, u);
                float f1 = fm(kc.f1k, mu);
                float f2 = fm(kc.f2k, fm(fm(mu, mu), mu));
                B.x = fa(B.x, fa(fm(f1, u.x), fm(f2, u.x)));
                B.y = fa(B.y, fa(fm(f1, u.y), fm(f2, u.y)));
                B.z = fa(B.z, fa(fm(f1, u.z), fm(f2, u.z)));
            } else {
                add_uniaxial(B, a.up, m0, I);
            }
        }
        if (!BAT && !UNI && a.cubic) add_cubic(B, a.cp, m0, I);  // engine/anisotropy.go:158
        if (a.zeeman) {
            if constexpr (BAT) {
                B.x = fa(B.x, ip->bext[0]);
                B.y = fa(B.y, ip->bext[1]);
                B.z = fa(B.z, ip->bext[2]);
            } else {
                const int r = UREG ? 0 : __ldg(a.regions + I);
                B.x = fa(B.x, __ldg(a.bext[0] + r));
                B.y = fa(B.y, __ldg(a.bext[1] + r));
                B.z = fa(B.z, __ldg(a.bext[2] + r));
            }
        }
        if (!BAT && !UNI && a.thermal) {  // engine/effectivefield.go:20-22 B_therm (temperature2.cl)
            const float sc = therm_scale(ctl->k2, amul(a.alpha, a.alpha_mul, I), amul(a.temp, a.temp_mul, I),
                                         inv_msat(a.Ms, a.Ms_mul, I));
            const f3 n = therm_normals(a.seed, ctl->nsteps, I);
            B.x = fa(B.x, fm(n.x, sc));
            B.y = fa(B.y, fm(n.y, sc));
            B.z = fa(B.z, fm(n.z, sc));
        }
        if (!UNI && a.beff) { a.beff[I] = B.x; a.beff[N + I] = B.y; a.beff[2 * N + I] = B.z; }
        f3 t;
        if (!UNI && !a.precess) t = llnoprecess(m0, B);
        else if (BAT || UNI || a.alpha_uniform) t = lltorque_g(m0, B, alpha_mul, kc.gilb);
        else t = lltorque(m0, B, amul(a.alpha, a.alpha_mul, I));
        // engine/torque.go:348-352 FreezeSpins (zeromask.cl)
        if (!BAT && !UNI && a.frozen && __ldg(a.frozen + (UREG ? 0 : __ldg(a.regions + I))) != 0.0f) t = f3{0.f, 0.f, 0.f};
        float* out = a.tau_direct ? a.tau_direct : ctl->k[a.out_slot];
        out[I] = t.x; out[N + I] = t.y; out[2 * N + I] = t.z;
        if constexpr (TAIL == kStageTail) stage_tail(in, ta, ctl, N, I, t);
        if constexpr (TAIL == kErrTail) err = err_tail(in, ta, t);
    }
    if constexpr (TAIL == kErrTail) err_finish(err, live, ta, ctl, gridDim.x * gridDim.y * (BAT ? a.g.Nz : gridDim.z));
}

// ---------------------------------------------------------------- stages
struct StageArgs {
    DevCtl* ctl;
    int N;
    int nterm;
    int src, dst;          // first term (coefficient 1) and result: 0 = ctl->m, 1 and 2 = ctl->mw[0] and [1]
    int slot[kMaxTerms];   // k slots of terms 1..nterm-1
    float c[kMaxTerms];    // float32 constants multiplying h (terms 1..)
    int normalize;
    int begin;             // the step's first kernel: start the step
    int only_if_accepted;  // the solution formed after the controller
    const float* vol;
};

// dst = normalize(src + sum_j (c_j h) k_j) with Madd<n> rounding
// (opencl/madd.go, madd<n>.cl) then normalize2.cl.  NT = number of terms.
template <int NT, bool BAT>
__global__ void __launch_bounds__(256) k_stage(StageArgs a) {
    DevCtl* ctl = a.ctl + (BAT ? blockIdx.y : 0);  // BAT: one grid row per instance
    pdl_wait();
    pdl_trigger();
    float h;
    if (a.begin) {
        if (blockIdx.x == 0 && threadIdx.x == 0) step_begin(ctl);
        if (!step_runs(ctl)) return;
        h = step_h(ctl);
    } else {
        if (!ctl->active) return;
        if (a.only_if_accepted && !ctl->accepted) return;
        h = ctl->h;
    }
    float fac[NT];
    const float* src[NT];
    fac[0] = 1.0f;
    src[0] = mbuf(ctl, a.src);
#pragma unroll
    for (int j = 1; j < NT; j++) {
        fac[j] = fm(a.c[j], h);
        src[j] = ctl->k[a.slot[j]];
    }
    float* dst = mbuf(ctl, a.dst);
    const int N = a.N;
    // one component of one cell from its NT source values (Madd<NT> order)
    auto comb = [&](const float (&x)[NT]) {
        if constexpr (NT == 3) {
            return fa(fm(fac[0], x[0]), fa(fm(fac[1], x[1]), fm(fac[2], x[2])));
        } else {
            float acc = fm(fac[0], x[0]);
#pragma unroll
            for (int j = 1; j < NT; j++) acc = fa(acc, fm(fac[j], x[j]));
            return acc;
        }
    };
    auto finish = [&](float (&v)[3], float w) {
        if (a.normalize) {
            f3 r = normalize_vol(f3{v[0], v[1], v[2]}, w);
            v[0] = r.x; v[1] = r.y; v[2] = r.z;
        }
    };
    // Four cells per iteration with 16-byte loads and stores where every
    // array allows it (N a multiple of 4, 16-byte aligned bases): four times
    // the bytes in flight per thread; each cell's arithmetic is unchanged.
    bool vec = (N & 3) == 0 && (reinterpret_cast<uintptr_t>(dst) & 15) == 0 &&
               (!a.vol || (reinterpret_cast<uintptr_t>(a.vol) & 15) == 0);
#pragma unroll
    for (int j = 0; j < NT; j++) vec = vec && (reinterpret_cast<uintptr_t>(src[j]) & 15) == 0;
    if (vec) {
        const int N4 = N >> 2;
        for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < N4; q += gridDim.x * blockDim.x) {
            float v[4][3];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                float4 x4[NT];
#pragma unroll
                for (int j = 0; j < NT; j++) x4[j] = reinterpret_cast<const float4*>(src[j] + (size_t)c * N)[q];
#pragma unroll
                for (int l = 0; l < 4; l++) {
                    float x[NT];
#pragma unroll
                    for (int j = 0; j < NT; j++) x[j] = l == 0 ? x4[j].x : l == 1 ? x4[j].y : l == 2 ? x4[j].z : x4[j].w;
                    v[l][c] = comb(x);
                }
            }
            const float4 w4 = a.vol ? reinterpret_cast<const float4*>(a.vol)[q] : make_float4(1.f, 1.f, 1.f, 1.f);
            finish(v[0], w4.x);
            finish(v[1], w4.y);
            finish(v[2], w4.z);
            finish(v[3], w4.w);
#pragma unroll
            for (int c = 0; c < 3; c++)
                reinterpret_cast<float4*>(dst + (size_t)c * N)[q] = make_float4(v[0][c], v[1][c], v[2][c], v[3][c]);
        }
        return;
    }
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        float v[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            float x[NT];
#pragma unroll
            for (int j = 0; j < NT; j++) x[j] = src[j][c * N + i];
            v[c] = comb(x);
        }
        finish(v, a.vol ? a.vol[i] : 1.0f);
        dst[i] = v[0]; dst[N + i] = v[1]; dst[2 * N + i] = v[2];
    }
}

// ---------------------------------------------------------------- error norms
struct ErrArgs {
    DevCtl* ctl;
    int N;
    int nterm;
    int slot[kMaxTerms];  // the last one's max norm is the torque of the new state (delM / k4 / dy)
    TailArgs ta;          // constants, Heun, controller
};

// kErrTail as a kernel of its own, four cells a thread.
template <int NT, bool HEUN, bool BAT>
__global__ void __launch_bounds__(256) k_err_norms(ErrArgs a) {
    DevCtl* ctl = a.ctl + (BAT ? blockIdx.y : 0);  // BAT: one grid row per instance
    pdl_wait();
    pdl_trigger();
    if (!ctl->active) return;
    const float* k[NT];
    float e[NT];
#pragma unroll
    for (int j = 0; j < NT; j++) {
        k[j] = ctl->k[a.slot[j]];
        e[j] = a.ta.c[j];
    }
    const float* dm = ctl->k[a.slot[NT - 1]];
    const int N = a.N;
    float me = 0.f, md = 0.f, mr = 0.f;
    int nan = 0;
    // one component of the error estimate of one cell (Madd<NT> order)
    auto comb = [&](const float (&x)[NT]) {
        if constexpr (HEUN) {
            return fs(x[0], x[1]);
        } else if constexpr (NT == 3) {
            return fa(fm(e[0], x[0]), fa(fm(e[1], x[1]), fm(e[2], x[2])));
        } else {
            float acc = fm(e[0], x[0]);
#pragma unroll
            for (int j = 1; j < NT; j++) acc = fa(acc, fm(e[j], x[j]));
            return acc;
        }
    };
    auto cell = [&](f3 E, f3 D) {
        float e2 = dot3(E, E), d2 = dot3(D, D);
        float en = __fsqrt_rn(e2), dn = __fsqrt_rn(d2);
        float r = dn == 0.0f ? 0.0f : fd(en, dn);
        nan |= (e2 != e2) | (d2 != d2);
        me = fmaxf(me, e2);
        md = fmaxf(md, d2);
        mr = fmaxf(mr, r);
    };
    // four cells per iteration with 16-byte loads where every array allows
    // it (the maxima do not depend on the order cells are visited in)
    bool vec = (N & 3) == 0 && (reinterpret_cast<uintptr_t>(dm) & 15) == 0;
#pragma unroll
    for (int j = 0; j < NT; j++) vec = vec && (reinterpret_cast<uintptr_t>(k[j]) & 15) == 0;
    if (vec) {
        const int N4 = N >> 2;
        for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < N4; q += gridDim.x * blockDim.x) {
            float E[4][3], D[4][3];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                float4 x4[NT];
#pragma unroll
                for (int j = 0; j < NT; j++) x4[j] = reinterpret_cast<const float4*>(k[j] + (size_t)c * N)[q];
                const float4 d4 = reinterpret_cast<const float4*>(dm + (size_t)c * N)[q];
                D[0][c] = d4.x; D[1][c] = d4.y; D[2][c] = d4.z; D[3][c] = d4.w;
#pragma unroll
                for (int l = 0; l < 4; l++) {
                    float x[NT];
#pragma unroll
                    for (int j = 0; j < NT; j++) x[j] = l == 0 ? x4[j].x : l == 1 ? x4[j].y : l == 2 ? x4[j].z : x4[j].w;
                    E[l][c] = comb(x);
                }
            }
#pragma unroll
            for (int l = 0; l < 4; l++) cell(f3{E[l][0], E[l][1], E[l][2]}, f3{D[l][0], D[l][1], D[l][2]});
        }
    } else {
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
            float Ec[3];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                float x[NT];
#pragma unroll
                for (int j = 0; j < NT; j++) x[j] = k[j][c * N + i];
                Ec[c] = comb(x);
            }
            cell(f3{Ec[0], Ec[1], Ec[2]}, f3{dm[i], dm[N + i], dm[2 * N + i]});
        }
    }
    err_finish(ErrMax{me, md, mr, nan}, true, a.ta, ctl, gridDim.x);
}

// ---------------------------------------------------------------- energies
// Per-term sums of dot(M_full, B_term) over the cells (engine/energy.go:51-69
// makeEdensAdder / dot, engine/anisotropy.go:164-216): M_full = Ms * m (* vol),
// the dot products in float32 as opencl.AddDotProduct/Dot form them, the sums
// accumulated in FP64 (compensated relative to the reference's float32
// reduction).  sums: [0] demag, [1] exchange (+DMI), [2] anisotropy from K1
// alone, [3] anisotropy from K2 alone, [4] Zeeman.
// the float32 dot products of cell I: [0] demag, [1] exchange (+DMI),
// [2] uniaxial anisotropy from K1 alone, [3] from K2 alone, [4] Zeeman,
// [5..7] cubic anisotropy from Kc1, Kc2, Kc3 alone, [8] thermal field
constexpr int kNE = 9;
__device__ __forceinline__ void energy_cell_terms(const LocalArgs& a, const float* __restrict__ vol, int I,
                                                  float t[kNE]) {
    const int N = a.N;
    const float* m = a.ctl->m;
    const float *mx = m, *my = m + N, *mz = m + 2 * N;
    const int ix = I % a.g.Nx, iy = (I / a.g.Nx) % a.g.Ny, iz = I / (a.g.Nx * a.g.Ny);
    const f3 m0 = ld3(mx, my, mz, I);
    const float ms = amul(a.Ms, a.Ms_mul, I);
    f3 Mf{fm(m0.x, ms), fm(m0.y, ms), fm(m0.z, ms)};
    if (vol) {
        const float w = __ldg(vol + I);
        Mf = f3{fm(Mf.x, w), fm(Mf.y, w), fm(Mf.z, w)};
    }
    for (int k = 0; k < kNE; k++) t[k] = 0.f;
    if (a.bd && !(a.nodemag && __ldg(a.nodemag + __ldg(a.regions + I)) != 0.0f))
        t[0] = dot3(Mf, f3{__ldg(a.bd + I), __ldg(a.bd + N + I), __ldg(a.bd + 2 * N + I)});
    if (!is0(m0)) {
        const int r0 = __ldg(a.regions + I);
        const f3 e = a.dbLUT ? dmibulk_sum(mx, my, mz, a.aLUT, a.dbLUT, a.regions, a.cx, a.cy, a.cz, a.g,
                                           a.openbc != 0, ix, iy, iz, m0, r0)
                   : a.dmi ? dmi_sum_lut(mx, my, mz, a.dl, a.regions, a.g, a.openbc != 0, ix, iy, iz, m0, r0)
                           : exchange_sum(mx, my, mz, a.aLUT, a.regions, a.wx, a.wy, a.wz, a.g, ix, iy, iz, m0, r0);
        const float inv = inv_msat(a.Ms, a.Ms_mul, I);
        t[1] = dot3(Mf, f3{fm(e.x, inv), fm(e.y, inv), fm(e.z, inv)});
    }
    if (a.anis) {
        UniaxParams p1 = a.up, p2 = a.up;
        p1.K2 = nullptr; p1.K2_mul = 0.f;
        p2.K1 = nullptr; p2.K1_mul = 0.f;
        f3 B1{0.f, 0.f, 0.f}, B2{0.f, 0.f, 0.f};
        add_uniaxial(B1, p1, m0, I);
        add_uniaxial(B2, p2, m0, I);
        t[2] = dot3(Mf, B1);
        t[3] = dot3(Mf, B2);
    }
    if (a.zeeman) {
        const int r = __ldg(a.regions + I);
        t[4] = dot3(Mf, f3{__ldg(a.bext[0] + r), __ldg(a.bext[1] + r), __ldg(a.bext[2] + r)});
    }
    if (a.thermal) {  // engine/temperature.go:21 Edens_therm: the field of the current step
        const float sc = therm_scale(a.ctl->k2, amul(a.alpha, a.alpha_mul, I), amul(a.temp, a.temp_mul, I),
                                     inv_msat(a.Ms, a.Ms_mul, I));
        const f3 n = therm_normals(a.seed, a.ctl->nsteps, I);
        t[8] = dot3(Mf, f3{fm(n.x, sc), fm(n.y, sc), fm(n.z, sc)});
    }
    if (a.cubic) {  // engine/anisotropy.go:191-206: each constant alone
        for (int k = 0; k < 3; k++) {
            CubicParams q = a.cp;
            if (k != 0) { q.K1 = nullptr; q.K1_mul = 0.f; }
            if (k != 1) { q.K2 = nullptr; q.K2_mul = 0.f; }
            if (k != 2) { q.K3 = nullptr; q.K3_mul = 0.f; }
            f3 Bc{0.f, 0.f, 0.f};
            add_cubic(Bc, q, m0, I);
            t[5 + k] = dot3(Mf, Bc);
        }
    }
}

__global__ void __launch_bounds__(256) k_energy_terms(LocalArgs a, const float* __restrict__ vol, double* sums) {
    __shared__ double sh[kNE][8];
    double acc[kNE] = {};
    for (int I = blockIdx.x * blockDim.x + threadIdx.x; I < a.N; I += gridDim.x * blockDim.x) {
        float t[kNE];
        energy_cell_terms(a, vol, I, t);
        for (int k = 0; k < kNE; k++) acc[k] += (double)t[k];
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int t = 0; t < kNE; t++) {
        double v = acc[t];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) sh[t][wid] = v;
    }
    __syncthreads();
    if (threadIdx.x < kNE) {
        double v = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) v += sh[threadIdx.x][w];
        atomicAdd(sums + threadIdx.x, v);
    }
}

// engine/demag.go:74-83: the demag convolution's volume with NoDemagSpins --
// a copy of the geometry (ones without one) zeroed where the region's value
// is non-zero (zeromask.cl), so those cells make no field
__global__ void k_nodemag_vol(const float* __restrict__ vol, const float* __restrict__ lut,
                              const uint8_t* __restrict__ regions, float* __restrict__ out, int N) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x)
        out[i] = __ldg(lut + __ldg(regions + i)) != 0.0f ? 0.0f : (vol ? __ldg(vol + i) : 1.0f);
}

// ---------------------------------------------------------------- host side
struct SimImpl {
    umag_sim_params p;
    umag_solver_params sp;
    int N;
    Mesh3 g;
    umag_demag* demag = nullptr;
    float* bufs = nullptr;        // 3 + 7 slots of 3N
    float* bd = nullptr;          // demag field 3N
    uint8_t* zero_regions = nullptr;
    float* dmi_pairs = nullptr;   // 7 x 32896 region-pair DMI coefficients
    float* demag_vol = nullptr;   // NoDemagSpins: geometry with the masked regions zeroed
    LocalConsts* kc_dev = nullptr;
    DevCtl* ctl = nullptr;        // device
    DevCtl* hctl = nullptr;       // pinned host mirror
    // run(): the controller records after the blocks of steps in flight
    DevCtl* hpoll = nullptr;      // pinned, 2
    cudaEvent_t polled[2] = {nullptr, nullptr};
    PassArgs pa{};
    LocalArgs la{};
    bool need_k1 = true;
    bool use_graph = true;
    int graph_steps = 16;
    cudaGraphExec_t gexec = nullptr;   // graph_steps steps
    cudaGraphExec_t gexec1 = nullptr;  // one step
    int launches_per_step = 0;
    double* esum = nullptr;            // energy term sums (kNE doubles)
    umag_tuning tune{{32, 8}, 256, 8, 4, 1};  // launch shapes (umag_sim_set_tuning)
    TileMaps tmaps{};                          // TMA maps of the three magnetisation buffers
    bool tile_ok = false;                      // the mesh and block shape allow tiles
    // batched ensemble class: nb same-size instances with uniform parameters
    int nb = 1;
    bool batched = false;
    InstParams* ip_dev = nullptr;
};

// stream the step/field launches go to: the library stream, or the stream of
// the ensemble class being captured
static thread_local cudaStream_t g_launch_stream = nullptr;
static cudaStream_t S() { return g_launch_stream ? g_launch_stream : ctx().stream; }
// Kernels of one simulation overlap the next one's start (common.cuh); those
// of an ensemble do not: waiting CTAs would hold the room that the other
// classes' kernels, on streams of their own, can use (48 films: 23.1 ms, 29.0 with
// it).  A general instance's demag passes still overlap among themselves.
static bool overlap(const SimImpl* s) { return !s->batched && !g_launch_stream; }
static unsigned ctl_grid(const SimImpl* s) { return (unsigned)((s->nb + 127) / 128); }

// the uniform-material instantiation: every term that it leaves out is off
static bool uniform_terms(const SimImpl* s) {
    const LocalArgs& la = s->la;
    return s->zero_regions && !la.nodemag && !la.dbLUT && !la.cubic && !la.thermal && !la.frozen && la.precess &&
           la.alpha_uniform && la.ms_uniform && (!la.anis || la.anis_uniform) && !la.openbc;
}
// Whether a step's stages and error estimate are formed in the torque kernel.
// It saves their launches and the torque's way through memory; but the
// kernel with maps and regions needs 64 registers for it, and holds fewer
// warps.  us a step of RK45DP, separate / fused kernels: uniform material,
// 256x256x4 258 / 253, 256x256x16 745 / 719, 512x512x32 6816 / 6747; region map
// and per-cell maps, 256x256x4 299 / 287, 256x256x16 851 / 867, 512x512x32
// 7771 / 8060.
static bool fuse_tails(const SimImpl* s) {
    if (!s->batched && s->tile_ok && s->tune.torque_tma && uniform_terms(s)) return true;
    return (long)s->N * s->nb <= (1L << 19);
}

// one torque evaluation of magnetisation buffer m_sel into ctl->k[slot] (or a
// direct buffer), and what follows it in the same kernel
template <int TAIL>
static cudaError_t torque_kernel(SimImpl* s, const LocalArgs& la, const TailArgs& ta, dim3 grd, dim3 blk, bool uni) {
    const bool tile = s->zero_regions && s->tile_ok && s->tune.torque_tma;
    auto k = s->batched ? k_local_torque<true, true, false, false, TAIL>
             : tile && uni ? k_local_torque<true, false, true, true, TAIL>
             : tile ? k_local_torque<true, false, true, false, TAIL>
             : s->zero_regions ? k_local_torque<true, false, false, false, TAIL>
                               : k_local_torque<false, false, false, false, TAIL>;
    const size_t sm = !s->batched && tile ? tile_bytes(blk.x, blk.y, s->g.Nz) + 128 : 0;
    return launch_pdl(overlap(s), k, grd, blk, sm, S(), la, s->tmaps, ta);
}
static int launch_torque(SimImpl* s, int m_sel, int slot, float* tau_direct, float* beff, int* nl,
                         const TailArgs& ta = TailArgs{}, bool early = false) {
    if (s->p.enable_demag) {
        PassArgs a = s->pa;
        a.m_sel = m_sel != 0;
        a.early = early;
        if (m_sel == 2) a.m_ind_w = &s->ctl->mw[1];
        if (s->batched) UMAG_TRY(demag_launch_batch(s->demag, a, s->nb, S(), overlap(s)));
        else UMAG_TRY(demag_launch(s->demag, a, S(), overlap(s)));
        if (nl) *nl += demag_launches(s->demag);
    }
    LocalArgs la = s->la;
    la.m_sel = m_sel;
    la.early = s->p.enable_demag;
    la.out_slot = slot;
    la.tau_direct = tau_direct;
    la.beff = beff;
    const int bx = s->tune.torque_block[0], by = s->tune.torque_block[1];
    dim3 blk(bx, by, 1), grd((s->g.Nx + bx - 1) / bx, (s->g.Ny + by - 1) / by, s->g.Nz * s->nb);
    const bool uni = uniform_terms(s) && !beff;
    if (ta.kind == kStageTail) UMAG_CUDA(torque_kernel<kStageTail>(s, la, ta, grd, blk, uni));
    else if (ta.kind == kErrTail) UMAG_CUDA(torque_kernel<kErrTail>(s, la, ta, grd, blk, uni));
    else UMAG_CUDA(torque_kernel<kNoTail>(s, la, ta, grd, blk, uni));
    if (nl) *nl += 1;
    return UMAG_OK;
}

static int launch_stage(SimImpl* s, int src, int dst, std::initializer_list<int> slots,
                        std::initializer_list<double> cs, bool normalize, bool begin, bool only_if_accepted, int* nl,
                        int last_slot = -1) {
    StageArgs a{};
    a.ctl = s->ctl;
    a.N = s->N;
    a.src = src;
    a.dst = dst;
    a.nterm = 1;
    for (int sl : slots) a.slot[a.nterm++] = sl;
    if (last_slot >= 0) a.slot[a.nterm++] = last_slot;
    int j = 1;
    for (double c : cs) a.c[j++] = (float)c;  // Go: untyped constant converted to float32
    a.normalize = normalize;
    a.begin = begin;
    a.only_if_accepted = only_if_accepted;
    a.vol = s->p.vol;
    const int th = s->tune.stage_threads;
    const dim3 g(s->batched ? (unsigned)((s->N + th - 1) / th) : (unsigned)grid_for(s->N, th, s->tune.stage_waves),
                 s->nb);
    void (*k)(StageArgs) = nullptr;
    switch (a.nterm) {
    case 2: k = s->batched ? k_stage<2, true> : k_stage<2, false>; break;
    case 3: k = s->batched ? k_stage<3, true> : k_stage<3, false>; break;
    case 4: k = s->batched ? k_stage<4, true> : k_stage<4, false>; break;
    case 5: k = s->batched ? k_stage<5, true> : k_stage<5, false>; break;
    case 6: k = s->batched ? k_stage<6, true> : k_stage<6, false>; break;
    default: return set_error(UMAG_E_ARG, "stage with %d terms", a.nterm);
    }
    UMAG_CUDA(launch_pdl(overlap(s), k, g, th, 0, S(), a));
    *nl += 1;
    return UMAG_OK;
}

// whether the kernel before an evaluation of a step leaves the controller record
// alone: all but the first one's, which starts the step
static bool later_eval(const SimImpl* s, int slot) { return slot != (s->sp.solver == 5 || s->sp.solver == 3 ? 1 : 0); }

// an evaluation into slot, then dst = normalize(m + h (sum_j cs_j k[slots_j] + cs_last k[slot]))
static int torque_stage(SimImpl* s, int m_sel, int slot, int dst, std::initializer_list<int> slots,
                        std::initializer_list<double> cs, int* nl, bool normalize = true) {
    if (!fuse_tails(s)) {
        UMAG_TRY(launch_torque(s, m_sel, slot, nullptr, nullptr, nl, TailArgs{}, later_eval(s, slot)));
        return launch_stage(s, 0, dst, slots, cs, normalize, false, false, nl, slot);
    }
    TailArgs t;
    t.kind = kStageTail;
    t.dst = dst;
    t.normalize = normalize;
    t.vol = s->p.vol;
    for (int sl : slots) t.slot[t.nk++] = sl;
    int j = 0;
    for (double c : cs) t.c[j++] = (float)c;  // Go: untyped constant converted to float32
    return launch_torque(s, m_sel, slot, nullptr, nullptr, nl, t, later_eval(s, slot));
}
// the step's last evaluation into slot, the error estimate
// sum_j es_j k[slots_j] + es_last k[slot] and the controller
static int torque_err(SimImpl* s, int m_sel, int slot, std::initializer_list<int> slots,
                      std::initializer_list<double> es, bool heun, const CtlArgs& q, int* nl) {
    TailArgs t;
    t.kind = kErrTail;
    t.heun = heun;
    t.ctl = q;
    for (int sl : slots) t.slot[t.nk++] = sl;
    int j = 0;
    for (double e : es) t.c[j++] = (float)e;
    if (fuse_tails(s)) return launch_torque(s, m_sel, slot, nullptr, nullptr, nl, t, later_eval(s, slot));
    UMAG_TRY(launch_torque(s, m_sel, slot, nullptr, nullptr, nl, TailArgs{}, later_eval(s, slot)));
    ErrArgs a{};
    a.ctl = s->ctl;
    a.N = s->N;
    for (int sl : slots) a.slot[a.nterm++] = sl;
    if (a.nterm == 0) a.slot[a.nterm++] = slot;  // Euler: the torque alone
    a.slot[a.nterm++] = slot;
    a.ta = t;
    const dim3 g(s->batched ? (unsigned)((s->N + 255) / 256) : (unsigned)grid_for(s->N, 256, s->tune.err_waves),
                 s->nb);
    void (*k)(ErrArgs) = nullptr;
    if (heun) k = s->batched ? k_err_norms<2, true, true> : k_err_norms<2, true, false>;
    else if (a.nterm == 2) k = s->batched ? k_err_norms<2, false, true> : k_err_norms<2, false, false>;
    else if (a.nterm == 4) k = s->batched ? k_err_norms<4, false, true> : k_err_norms<4, false, false>;
    else if (a.nterm == 6) k = s->batched ? k_err_norms<6, false, true> : k_err_norms<6, false, false>;
    else return set_error(UMAG_E_ARG, "error combination with %d terms", a.nterm);
    UMAG_CUDA(launch_pdl(overlap(s), k, g, 256, 0, S(), a));
    *nl += 1;
    return UMAG_OK;
}

// Slots: k[0] = k1 (FSAL), k[1..6] = k2..k7 buffers.  Each evaluation's kernel
// writes the next stage's magnetisation to the working buffer that it does not
// read (1 and 2 in turn).
static int launch_step(SimImpl* s, int* nl) {
    auto begin = [&]() -> int {
        UMAG_CUDA(launch_pdl(overlap(s), k_step_begin, ctl_grid(s), 128, 0, S(), s->ctl, s->nb));
        *nl += 1;
        return UMAG_OK;
    };
    switch (s->sp.solver) {
    case 5: {  // engine/rk45dp.go:52-97
        UMAG_TRY(launch_stage(s, 0, 1, {0}, {1. / 5.}, true, true, false, nl));
        UMAG_TRY(torque_stage(s, 1, 1, 2, {0}, {3. / 40., 9. / 40.}, nl));
        UMAG_TRY(torque_stage(s, 2, 2, 1, {0, 1}, {44. / 45., -56. / 15., 32. / 9.}, nl));
        UMAG_TRY(torque_stage(s, 1, 3, 2, {0, 1, 2}, {19372. / 6561., -25360. / 2187., 64448. / 6561., -212. / 729.}, nl));
        UMAG_TRY(torque_stage(s, 2, 4, 1, {0, 1, 2, 3},
                              {9017. / 3168., -355. / 33., 46732. / 5247., 49. / 176., -5103. / 18656.}, nl));
        UMAG_TRY(torque_stage(s, 1, 5, 2, {0, 2, 3, 4},
                              {35. / 384., 500. / 1113., 125. / 192., -2187. / 6784., 11. / 84.}, nl));
        // rk45dp.go:95 weight differences, as exact rationals rounded to float32
        return torque_err(s, 2, 6, {0, 2, 3, 4, 5},
                          {71. / 57600., -71. / 16695., 71. / 1920., -17253. / 339200., 22. / 525., -1. / 40.}, false,
                          CtlArgs{0, 5, 6, 6, 0, 6, 2, 0}, nl);
    }
    case 3: {  // engine/rk23.go:58-83
        UMAG_TRY(launch_stage(s, 0, 1, {0}, {1. / 2.}, true, true, false, nl));
        UMAG_TRY(torque_stage(s, 1, 1, 2, {}, {3. / 4.}, nl));
        UMAG_TRY(torque_stage(s, 2, 2, 1, {0, 1}, {2. / 9., 1. / 3., 4. / 9.}, nl));
        return torque_err(s, 1, 3, {0, 1, 2}, {5. / 72., -1. / 12., -1. / 9., 1. / 8.}, false,
                          CtlArgs{0, 3, 4, 3, 0, 3, 1, 0}, nl);
    }
    case 2: {  // engine/heun.go:15-59
        UMAG_TRY(begin());
        UMAG_TRY(torque_stage(s, 0, 0, 1, {}, {1.0}, nl, false));  // dy0; y = y + dt*dy0
        UMAG_TRY(torque_err(s, 1, 1, {0}, {}, true, CtlArgs{2, 2, 3, -1, -1, 2, 1, 0}, nl));  // dy; |dy0 - dy|
        // accepted: y = y + 0.5 dt dy - 0.5 dt dy0, normalised (heun.go:45-46)
        return launch_stage(s, 0, 0, {1, 0}, {0.5, -0.5}, true, false, true, nl);
    }
    case 1: {  // engine/euler.go:11-36
        UMAG_TRY(begin());
        UMAG_TRY(torque_err(s, 0, 0, {}, {}, true, CtlArgs{3, 1, 1, -1, -1, 1, 1, 0}, nl));  // dy0, max |dy0|
        // y = y + dt*dy0 (Madd2), normalised (euler.go:33-34)
        return launch_stage(s, 1, 0, {0}, {1.0}, true, false, true, nl);
    }
    case 4: {  // engine/rk4.go:11-69
        UMAG_TRY(begin());
        UMAG_TRY(torque_stage(s, 0, 0, 1, {}, {1. / 2.}, nl));
        UMAG_TRY(torque_stage(s, 1, 1, 2, {}, {1. / 2.}, nl));
        UMAG_TRY(torque_stage(s, 2, 2, 1, {}, {1.}, nl));
        UMAG_TRY(torque_err(s, 1, 3, {0}, {1., -1.}, false, CtlArgs{1, 4, 5, -1, -1, 4, 1, 1}, nl));
        return launch_stage(s, 1, 0, {0, 1, 2, 3}, {1. / 6., 1. / 3., 1. / 3., 1. / 6.}, true, false, true, nl);
    }
    default:
        return set_error(UMAG_E_ARG, "unknown solver %d", s->sp.solver);
    }
}

static int sync_ctl_to_host(SimImpl* s) {
    UMAG_CUDA(cudaMemcpyAsync(s->hctl, s->ctl, sizeof(DevCtl) * s->nb, cudaMemcpyDeviceToHost, S()));
    UMAG_CUDA(cudaStreamSynchronize(S()));
    return UMAG_OK;
}
static int push_ctl(SimImpl* s) {
    UMAG_CUDA(cudaMemcpyAsync(s->ctl, s->hctl, sizeof(DevCtl) * s->nb, cudaMemcpyHostToDevice, S()));
    UMAG_CUDA(cudaStreamSynchronize(S()));
    return UMAG_OK;
}

// FSAL k1 of the current state, before the first step of a run
// (engine/rk45dp.go:26-29; RunWhile frees the stepper, engine/run.go:207)
static int ensure_k1(SimImpl* s) {
    if (!s->need_k1) return UMAG_OK;
    if (s->sp.solver == 5 || s->sp.solver == 3) {
        UMAG_TRY(sync_ctl_to_host(s));
        for (int b = 0; b < s->nb; b++) s->hctl[b].active = 1;
        UMAG_TRY(push_ctl(s));
        UMAG_TRY(launch_torque(s, 0, 0, nullptr, nullptr, nullptr));
        UMAG_TRY(sync_ctl_to_host(s));
        for (int b = 0; b < s->nb; b++) s->hctl[b].nevals += 1;
        UMAG_TRY(push_ctl(s));
    }
    s->need_k1 = false;
    return UMAG_OK;
}

static void drop_graph(SimImpl* s) {
    if (s->gexec) cudaGraphExecDestroy(s->gexec);
    if (s->gexec1) cudaGraphExecDestroy(s->gexec1);
    s->gexec = nullptr;
    s->gexec1 = nullptr;
}

// capture `steps` steps into *out
static int capture_steps(SimImpl* s, int steps, cudaGraphExec_t* out) {
    cudaGraph_t graph;
    UMAG_CUDA(cudaStreamBeginCapture(S(), cudaStreamCaptureModeThreadLocal));
    int nl = 0;
    int st = UMAG_OK;
    for (int i = 0; i < steps && st == UMAG_OK; i++) st = launch_step(s, &nl);
    cudaError_t e = cudaStreamEndCapture(S(), &graph);
    if (st != UMAG_OK) return st;
    if (e != cudaSuccess) return set_error(UMAG_E_CUDA, "graph capture: %s", cudaGetErrorString(e));
    e = cudaGraphInstantiate(out, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) return set_error(UMAG_E_CUDA, "graph instantiate: %s", cudaGetErrorString(e));
    return UMAG_OK;
}

// n steps with the stop time already in ctl: graphs of graph_steps steps,
// the remainder from a one-step graph
static int run_steps(SimImpl* s, long long n) {
    UMAG_TRY(ensure_k1(s));
    if (s->use_graph) {
        if (n >= s->graph_steps) {
            if (!s->gexec) UMAG_TRY(capture_steps(s, s->graph_steps, &s->gexec));
            for (; n >= s->graph_steps; n -= s->graph_steps) UMAG_CUDA(cudaGraphLaunch(s->gexec, S()));
        }
        if (n > 0) {
            if (!s->gexec1) UMAG_TRY(capture_steps(s, 1, &s->gexec1));
            for (; n > 0; n--) UMAG_CUDA(cudaGraphLaunch(s->gexec1, S()));
        }
        return UMAG_OK;
    }
    for (long long i = 0; i < n; i++) {
        int nl = 0;
        UMAG_TRY(launch_step(s, &nl));
    }
    return UMAG_OK;
}

// Tensor maps for the magnetisation tiles of the torque kernel (tile.cuh),
// when the mesh allows them: region-free, non-periodic, not batched, no bulk
// DMI, Nx a multiple of 4 (row strides and buffer offsets in 16-byte units),
// and a box of at most 256 elements per dimension.
static void tile_setup(SimImpl* s) {
    s->tile_ok = false;
    const int bx = s->tune.torque_block[0], by = s->tune.torque_block[1];
    if (s->batched || !s->zero_regions || s->g.pbc != 0 || s->la.dbLUT || s->g.Nx % 4 != 0) return;
    if (tile_pitch(bx) > 256 || tile_rows(by) > 256) return;
    EncodeTiledFn fn = encode_tiled();
    if (!fn) return;
    const cuuint64_t dims[4] = {(cuuint64_t)s->g.Nx, (cuuint64_t)s->g.Ny, (cuuint64_t)s->g.Nz, 3};
    const cuuint64_t strides[3] = {sizeof(float) * (cuuint64_t)s->g.Nx,
                                   sizeof(float) * (cuuint64_t)s->g.Nx * s->g.Ny, sizeof(float) * (cuuint64_t)s->N};
    const cuuint32_t box[4] = {(cuuint32_t)tile_pitch(bx), (cuuint32_t)tile_rows(by),
                               (cuuint32_t)(s->g.Nz > 1 ? 3 : 1), 3};
    const cuuint32_t es[4] = {1, 1, 1, 1};
    for (int b = 0; b < 3; b++) {
        float* base = s->bufs + (size_t)b * 3 * s->N;
        if (reinterpret_cast<uintptr_t>(base) % 16 != 0) return;
        if (fn(&s->tmaps.map[b], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, base, dims, strides, box, es,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return;
    }
    s->tile_ok = true;
}

// The local-term arguments that follow from the material parameters in s->p
// (and the uniform factors evaluated from them); run at creation and again
// whenever a parameter is reassigned.
static int local_from_params(SimImpl* s) {
    const umag_sim_params* p = &s->p;
    LocalArgs& la = s->la;
    la.aLUT = p->aLUT;
    la.dLUT = p->dLUT;
    la.regions = s->p.regions;
    la.wx = (float)(2 / (p->cell[0] * p->cell[0]));
    la.wy = (float)(2 / (p->cell[1] * p->cell[1]));
    la.wz = (float)(2 / (p->cell[2] * p->cell[2]));
    la.cx = (float)p->cell[0]; la.cy = (float)p->cell[1]; la.cz = (float)p->cell[2];
    la.dmi = p->dLUT != nullptr;
    la.openbc = p->openbc;
    la.anis = (p->Ku1 != nullptr || p->Ku1_mul != 0.f || p->Ku2 != nullptr || p->Ku2_mul != 0.f);
    la.up = UniaxParams{p->Ms, p->Ku1, p->Ku2, p->anisU[0], p->anisU[1], p->anisU[2],
                        p->Ms_mul, p->Ku1_mul, p->Ku2_mul, p->anisU_mul[0], p->anisU_mul[1], p->anisU_mul[2]};
    la.zeeman = p->bextLUT[0] != nullptr;
    for (int i = 0; i < 3; i++) la.bext[i] = p->bextLUT[i];
    la.alpha = p->alpha;
    la.alpha_mul = p->alpha_mul;
    la.precess = p->precess;
    la.frozen = p->frozen_lut;
    la.nodemag = p->enable_demag ? p->nodemag_lut : nullptr;
    la.cubic = (p->Kc1 != nullptr || p->Kc1_mul != 0.f || p->Kc2 != nullptr || p->Kc2_mul != 0.f ||
                p->Kc3 != nullptr || p->Kc3_mul != 0.f);
    la.cp = CubicParams{p->Ms, p->Kc1, p->Kc2, p->Kc3, {p->anisC1[0], p->anisC1[1], p->anisC1[2]},
                        {p->anisC2[0], p->anisC2[1], p->anisC2[2]}, p->Ms_mul, p->Kc1_mul, p->Kc2_mul, p->Kc3_mul,
                        {p->anisC1_mul[0], p->anisC1_mul[1], p->anisC1_mul[2]},
                        {p->anisC2_mul[0], p->anisC2_mul[1], p->anisC2_mul[2]}};
    la.dbLUT = p->dbulkLUT;
    la.thermal = (p->temp != nullptr || p->temp_mul != 0.f);
    la.temp = p->temp;
    la.temp_mul = p->temp_mul;
    la.seed = p->therm_seed;
    la.Ms = p->Ms;
    la.Ms_mul = p->Ms_mul;
    la.ms_uniform = p->Ms == nullptr;
    la.alpha_uniform = p->alpha == nullptr;
    la.anis_uniform = p->Ms == nullptr && p->Ku1 == nullptr && p->Ku2 == nullptr && p->anisU[0] == nullptr &&
                      p->anisU[1] == nullptr && p->anisU[2] == nullptr;
    {  // uniform factors, evaluated on the device (bit-identical to the per-cell path)
        if (!s->kc_dev && cudaMalloc(&s->kc_dev, sizeof(LocalConsts)) != cudaSuccess)
            return set_error(UMAG_E_NOMEM, "consts");
        k_local_consts<<<1, 1, 0, S()>>>(la, s->kc_dev);
        if (cudaMemcpyAsync(&la.kc, s->kc_dev, sizeof(LocalConsts), cudaMemcpyDeviceToHost, S()) != cudaSuccess ||
            cudaStreamSynchronize(S()) != cudaSuccess)
            return set_error(UMAG_E_CUDA, "uniform constants");
    }
    if (s->demag) {
        s->pa.Ms = p->Ms;
        s->pa.Ms_mul = p->Ms_mul;
    }
    return UMAG_OK;
}

int sim_new(const umag_sim_params* p, const umag_solver_params* sp, umag_sim** out) {
    UMAG_TRY(ensure_init());
    UMAG_REQUIRE(p && sp && out, "NULL argument");
    UMAG_REQUIRE(p->N[0] > 0 && p->N[1] > 0 && p->N[2] > 0, "bad mesh size");
    UMAG_REQUIRE(p->aLUT != nullptr, "aLUT (exchange LUT) is required");
    UMAG_REQUIRE(sp->solver >= 1 && sp->solver <= 5,
                 "solver must be 1 (Euler), 2 (Heun), 3 (RK23), 4 (RK4) or 5 (RK45DP)");
    UMAG_REQUIRE(p->pbc[0] >= 0 && p->pbc[1] >= 0 && p->pbc[2] >= 0, "PBC repetitions must be non-negative");
    // engine/exchange.go:62-63
    UMAG_REQUIRE(!(p->dLUT && p->dbulkLUT), "Cannot have induced and interfacial DMI at the same time");
    SimImpl* s = new SimImpl();
    s->p = *p;
    s->sp = *sp;
    s->N = p->N[0] * p->N[1] * p->N[2];
    // data/mesh.go PBC_code: the stencils wrap along periodic axes
    s->g = Mesh3{p->N[0], p->N[1], p->N[2], (p->pbc[0] ? 1 : 0) | (p->pbc[1] ? 2 : 0) | (p->pbc[2] ? 4 : 0)};
    int st = UMAG_OK;
    size_t b3 = sizeof(float) * 3 * (size_t)s->N;
    auto fail = [&](int code) { sim_free(reinterpret_cast<umag_sim*>(s)); return code; };
    if (cudaMalloc(&s->bufs, b3 * 10) != cudaSuccess) return fail(set_error(UMAG_E_NOMEM, "state buffers"));
    if (cudaMemsetAsync(s->bufs, 0, b3 * 10, S()) != cudaSuccess) return fail(set_error(UMAG_E_CUDA, "state buffers"));
    if (!p->regions) {
        if (cudaMalloc(&s->zero_regions, s->N) != cudaSuccess) return fail(set_error(UMAG_E_NOMEM, "regions"));
        if (cudaMemsetAsync(s->zero_regions, 0, s->N, S()) != cudaSuccess) return fail(set_error(UMAG_E_CUDA, "regions"));
        s->p.regions = s->zero_regions;
    }
    if (p->enable_demag) {
        const int pbc[3] = {p->pbc[0], p->pbc[1], p->pbc[2]};
        if (p->demag_kernel == 1)
            st = demag_new_brute(p->N[0], p->N[1], p->N[2], pbc, p->cell[0], p->cell[1], p->cell[2],
                                 p->demag_accuracy > 0 ? p->demag_accuracy : 6.0, &s->demag);
        else
            st = demag_new_newell(p->N[0], p->N[1], p->N[2], pbc, p->cell[0], p->cell[1], p->cell[2],
                                  p->asymptotic_radius > 0 ? p->asymptotic_radius : 32, 0, &s->demag);
        if (st != UMAG_OK) return fail(st);
        if (cudaMalloc(&s->bd, b3) != cudaSuccess) return fail(set_error(UMAG_E_NOMEM, "demag field"));
    }
    if (cudaMalloc(&s->ctl, sizeof(DevCtl)) != cudaSuccess) return fail(set_error(UMAG_E_NOMEM, "ctl"));
    if (cudaMallocHost(&s->hctl, sizeof(DevCtl)) != cudaSuccess) return fail(set_error(UMAG_E_NOMEM, "ctl host"));
    if (cudaMallocHost(&s->hpoll, 2 * sizeof(DevCtl)) != cudaSuccess) return fail(set_error(UMAG_E_NOMEM, "ctl host"));
    for (auto& e : s->polled)
        if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess)
            return fail(set_error(UMAG_E_CUDA, "poll events"));
    DevCtl& c = *s->hctl;
    memset(&c, 0, sizeof(c));
    c.m = s->bufs;
    for (int i = 0; i < 2; i++) c.mw[i] = s->bufs + (1 + i) * 3 * (size_t)s->N;
    for (int i = 0; i < 7; i++) c.k[i] = s->bufs + (3 + i) * 3 * (size_t)s->N;
    c.dt = sp->dt;
    c.alarm = 0.0;
    c.stop = INFINITY;
    c.max_err = sp->max_err; c.rel_err = sp->rel_err; c.min_dt = sp->min_dt; c.max_dt = sp->max_dt;
    c.fix_dt = sp->fix_dt; c.headroom = sp->headroom; c.min_slope = sp->min_slope; c.gamma = sp->gamma_ll;
    c.active = 1;
    if (p->temp != nullptr || p->temp_mul != 0.f) {  // engine/temperature.go:111 (cellVolume: c0 c1 c2)
        c.therm_gv = sp->gamma_ll * (p->cell[0] * p->cell[1] * p->cell[2]);
        const double dt0 = sp->fix_dt != 0 ? sp->fix_dt : sp->dt;
        c.k2 = (float)(2 * kBoltzmann / (c.therm_gv * dt0));
    }
    st = push_ctl(s);
    if (st != UMAG_OK) return fail(st);
    // pass / local arguments
    if (s->demag) {
        fill_pass_args(s->demag, s->pa);
        s->pa.m_ind = &s->ctl->m;
        s->pa.m_ind_w = &s->ctl->mw[0];
        s->pa.active = &s->ctl->active;
        s->pa.fault = &s->ctl->status;
        s->pa.vol = p->vol;
        s->pa.Ms = p->Ms;
        s->pa.Ms_mul = p->Ms_mul;
        s->pa.ncell = s->N;
        for (int i = 0; i < 3; i++) s->pa.B[i] = s->bd + (size_t)i * s->N;
        if (p->nodemag_lut) {  // engine/demag.go:67-98 setMaskedDemagField
            if (cudaMalloc(&s->demag_vol, sizeof(float) * s->N) != cudaSuccess)
                return fail(set_error(UMAG_E_NOMEM, "NoDemagSpins volume"));
            k_nodemag_vol<<<grid_for(s->N, 256), 256, 0, S()>>>(p->vol, p->nodemag_lut, s->p.regions, s->demag_vol,
                                                                s->N);
            if (cudaStreamSynchronize(S()) != cudaSuccess) return fail(set_error(UMAG_E_CUDA, "NoDemagSpins volume"));
            s->pa.vol = s->demag_vol;
        }
    }
    LocalArgs& la = s->la;
    la.g = s->g;
    la.N = s->N;
    la.ctl = s->ctl;
    la.bd = s->bd;
    st = local_from_params(s);
    if (st != UMAG_OK) return fail(st);
    for (int i = 0; i < 2; i++) la.mbuf[i] = s->bufs + (1 + i) * 3 * (size_t)s->N;
    // default launch shapes for small meshes: enough CTAs to reach most SMs
    // (the autotuner may choose others; results do not depend on them)
    if ((long)((s->g.Nx + 31) / 32) * ((s->g.Ny + 7) / 8) * s->g.Nz < ctx().sm_count) s->tune.torque_block[1] = 2;
    if ((long)s->N < (long)ctx().sm_count * 256) s->tune.stage_threads = 64;
    tile_setup(s);
    if (la.dmi) {
        const int np = 256 * 257 / 2;
        if (cudaMalloc(&s->dmi_pairs, sizeof(float) * 7 * np) != cudaSuccess)
            return fail(set_error(UMAG_E_NOMEM, "DMI pair table"));
        float* t = s->dmi_pairs;
        la.dl = DmiPairLut{t, t + np, t + 2 * np, t + 3 * np, t + 4 * np, t + 5 * np, t + 6 * np};
        k_dmi_pairs<<<grid_for(np, 256), 256, 0, S()>>>(p->aLUT, p->dLUT, la.cx, la.cy, la.cz, t, t + np, t + 2 * np,
                                                        t + 3 * np, t + 4 * np, t + 5 * np, t + 6 * np, np);
        if (cudaStreamSynchronize(S()) != cudaSuccess) return fail(set_error(UMAG_E_CUDA, "DMI pair table"));
    }
    if (la.zeeman && (!p->bextLUT[1] || !p->bextLUT[2])) return fail(set_error(UMAG_E_ARG, "bextLUT needs 3 arrays"));
    int nl = 0;
    // count launches of one step (not enqueued: measured on a dry capture below)
    s->launches_per_step = 0;
    {
        cudaGraph_t graph;
        if (cudaStreamBeginCapture(S(), cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
            st = launch_step(s, &nl);
            cudaStreamEndCapture(S(), &graph);
            cudaGraphDestroy(graph);
            if (st != UMAG_OK) return fail(st);
            s->launches_per_step = nl;
        }
    }
    *out = reinterpret_cast<umag_sim*>(s);
    return UMAG_OK;
}

int sim_free(umag_sim* h) {
    SimImpl* s = reinterpret_cast<SimImpl*>(h);
    if (!s) return UMAG_OK;
    cudaStreamSynchronize(S());
    drop_graph(s);
    if (s->demag) demag_free(s->demag);
    cudaFree(s->bufs);
    cudaFree(s->bd);
    cudaFree(s->zero_regions);
    cudaFree(s->dmi_pairs);
    cudaFree(s->demag_vol);
    cudaFree(s->kc_dev);
    cudaFree(s->esum);
    cudaFree(s->ctl);
    if (s->hctl) cudaFreeHost(s->hctl);
    if (s->hpoll) cudaFreeHost(s->hpoll);
    for (auto e : s->polled)
        if (e) cudaEventDestroy(e);
    delete s;
    return UMAG_OK;
}

// normalise = 0 restores a state read by sim_get_m exactly (normalising an
// already normalised float32 vector may change its last bit)
int sim_set_m(umag_sim* h, const float* mx, const float* my, const float* mz, int normalise) {
    SimImpl* s = reinterpret_cast<SimImpl*>(h);
    UMAG_REQUIRE(s && mx && my && mz, "NULL argument");
    UMAG_TRY(sync_ctl_to_host(s));
    float* m = s->hctl->m;
    size_t b = sizeof(float) * s->N;
    UMAG_CUDA(cudaMemcpyAsync(m, mx, b, cudaMemcpyDeviceToDevice, S()));
    UMAG_CUDA(cudaMemcpyAsync(m + s->N, my, b, cudaMemcpyDeviceToDevice, S()));
    UMAG_CUDA(cudaMemcpyAsync(m + 2 * s->N, mz, b, cudaMemcpyDeviceToDevice, S()));
    // engine/magnetization.go:34 normalize() (normalize2.cl)
    if (normalise) UMAG_TRY(normalize(m, m + s->N, m + 2 * s->N, s->p.vol, s->N));
    else UMAG_CUDA(cudaStreamSynchronize(S()));
    s->need_k1 = true;
    return UMAG_OK;
}

int sim_m_ptrs(umag_sim* h, float** m3) {
    SimImpl* s = reinterpret_cast<SimImpl*>(h);
    UMAG_REQUIRE(s && m3, "NULL argument");
    UMAG_TRY(sync_ctl_to_host(s));
    for (int c = 0; c < 3; c++) m3[c] = s->hctl->m + (size_t)c * s->N;
    return UMAG_OK;
}

int sim_get_m(umag_sim* h, float* mx, float* my, float* mz) {
    SimImpl* s = reinterpret_cast<SimImpl*>(h);
    UMAG_REQUIRE(s && mx && my && mz, "NULL argument");
    float* m3[3];
    UMAG_TRY(sim_m_ptrs(h, m3));
    size_t b = sizeof(float) * s->N;
    float* dst[3] = {mx, my, mz};
    for (int c = 0; c < 3; c++) UMAG_CUDA(cudaMemcpyAsync(dst[c], m3[c], b, cudaMemcpyDefault, S()));
    UMAG_CUDA(cudaStreamSynchronize(S()));
    return UMAG_OK;
}

int sim_torque(umag_sim* h, float* tx, float* ty, float* tz, float* bx, float* by, float* bz) {
    SimImpl* s = reinterpret_cast<SimImpl*>(h);
    UMAG_REQUIRE(s && tx && ty && tz, "NULL argument");
    UMAG_REQUIRE(ty == tx + s->N && tz == tx + 2 * s->N, "torque arrays must be one contiguous 3N buffer");
    if (bx) UMAG_REQUIRE(by == bx + s->N && bz == bx + 2 * s->N, "B_eff arrays must be one contiguous 3N buffer");
    UMAG_TRY(sync_ctl_to_host(s));
    s->hctl->active = 1;
    UMAG_TRY(push_ctl(s));
    UMAG_TRY(launch_torque(s, 0, 0, tx, bx, nullptr));
    UMAG_CUDA(cudaStreamSynchronize(S()));
    return UMAG_OK;
}

int sim_steps(umag_sim* h, int n) {
    SimImpl* s = reinterpret_cast<SimImpl*>(h);
    UMAG_REQUIRE(s && n >= 0, "bad argument");
    UMAG_TRY(sync_ctl_to_host(s));
    s->hctl->stop = INFINITY;
    UMAG_TRY(push_ctl(s));
    return run_steps(s, n);
}

// Steps from record c to its stop time, if the time step stayed as it is.
static long long steps_left(const DevCtl& c) {
    if (!(c.t < c.stop) || c.status != 0) return 0;
    const double n = std::ceil((c.stop - c.t) / c.dt);
    return n >= 1 ? (n < 1e9 ? (long long)n : 1000000000LL) : 1;
}

// Steps queued past the stop time do nothing but cost their launches (a tenth
// of the run for 27 steps of 256x256x16 queued as 64), and waiting for each
// step would leave gaps.  So blocks of steps are queued as far as the last
// record says that they are needed, two blocks ahead at most: first 8 steps
// (the time step still grows), then 16.
int sim_run(umag_sim* h, double seconds, int chunk, long long max_steps) {
    SimImpl* s = reinterpret_cast<SimImpl*>(h);
    UMAG_REQUIRE(s && seconds >= 0, "bad argument");
    if (chunk <= 0) chunk = 64;
    UMAG_TRY(sync_ctl_to_host(s));
    double stop = s->hctl->t + seconds;
    s->hctl->stop = stop;
    s->hctl->alarm = stop;  // engine/run.go:190-195: adaptDt must not cross it
    UMAG_TRY(push_ctl(s));
    s->need_k1 = true;      // RunWhile frees the stepper (engine/run.go:207)
    if (max_steps > 0) UMAG_TRY(ensure_k1(s));
    long long queued = 0, known = 0, ends[2] = {0, 0}, left = steps_left(*s->hctl);
    int in_flight = 0, oldest = 0;
    while (left > 0) {
        long long n = std::min(left - (queued - known), max_steps - queued);
        if (n > 0 && in_flight < 2) {
            n = std::min(n, (long long)std::min(chunk, known > 0 && n >= 32 ? 16 : 8));
            UMAG_TRY(run_steps(s, n));
            queued += n;
            const int q = (oldest + in_flight++) % 2;
            ends[q] = queued;
            UMAG_CUDA(cudaMemcpyAsync(s->hpoll + q, s->ctl, sizeof(DevCtl), cudaMemcpyDeviceToHost, S()));
            UMAG_CUDA(cudaEventRecord(s->polled[q], S()));
            continue;
        }
        if (in_flight == 0) break;  // max_steps
        UMAG_CUDA(cudaEventSynchronize(s->polled[oldest]));
        left = steps_left(s->hpoll[oldest]);
        known = ends[oldest];
        oldest ^= 1;
        in_flight--;
    }
    UMAG_TRY(sync_ctl_to_host(s));
    if (s->hctl->status != 0) return set_error(UMAG_E_SOLVER, "solver failure code %d at t=%g", s->hctl->status,
                                               s->hctl->t);
    return UMAG_OK;
}

// test hook: the device-side status word set as a kernel whose bounded wait
// gave up would set it (the host-side checks then see it)
int sim_plant_status(umag_sim* h, int code) {
    SimImpl* s = reinterpret_cast<SimImpl*>(h);
    UMAG_REQUIRE(s, "NULL simulation");
    UMAG_CUDA(cudaStreamSynchronize(S()));
    UMAG_CUDA(cudaMemcpyAsync(reinterpret_cast<char*>(s->ctl) + offsetof(DevCtl, status), &code, sizeof(int),
                              cudaMemcpyHostToDevice, S()));
    UMAG_CUDA(cudaStreamSynchronize(S()));
    return UMAG_OK;
}

int sim_get_state(umag_sim* h, umag_solver_state* st) {
    SimImpl* s = reinterpret_cast<SimImpl*>(h);
    UMAG_REQUIRE(s && st, "NULL argument");
    UMAG_TRY(sync_ctl_to_host(s));
    const DevCtl& c = *s->hctl;
    st->time = c.t; st->dt = c.dt; st->last_err = c.last_err; st->peak_err = c.peak_err;
    st->last_torque = c.last_torque; st->nsteps = c.nsteps; st->nundone = c.nundone; st->nevals = c.nevals;
    st->status = c.status;
    return UMAG_OK;
}

int sim_set_time(umag_sim* h, double t, double dt) {
    SimImpl* s = reinterpret_cast<SimImpl*>(h);
    UMAG_REQUIRE(s, "NULL argument");
    UMAG_TRY(sync_ctl_to_host(s));
    s->hctl->t = t;
    if (dt > 0) s->hctl->dt = dt;
    return push_ctl(s);
}

int sim_average_m(umag_sim* h, double avg[3]) {
    SimImpl* s = reinterpret_cast<SimImpl*>(h);
    UMAG_REQUIRE(s && avg, "NULL argument");
    float* m3[3];
    UMAG_TRY(sim_m_ptrs(h, m3));
    // engine/average.go:29-40: sum (or vol-weighted sum) over the magnet / cell count
    double ncell = (double)s->N;
    if (s->p.vol) UMAG_TRY(sum_dot(s->p.vol, nullptr, s->N, &ncell));
    for (int c = 0; c < 3; c++) {
        double v;
        UMAG_TRY(sum_dot(m3[c], s->p.vol, s->N, &v));
        avg[c] = v / ncell;
    }
    return UMAG_OK;
}

int sim_use_graph(umag_sim* h, int enable, int steps) {
    SimImpl* s = reinterpret_cast<SimImpl*>(h);
    UMAG_REQUIRE(s, "NULL argument");
    s->use_graph = enable != 0;
    if (steps > 0 && steps != s->graph_steps) {
        s->graph_steps = steps;
        drop_graph(s);
    }
    return UMAG_OK;
}

int sim_torque_evals(umag_sim* h, int n) {
    SimImpl* s = reinterpret_cast<SimImpl*>(h);
    UMAG_REQUIRE(s && n >= 0, "bad argument");
    UMAG_TRY(ensure_k1(s));
    UMAG_TRY(sync_ctl_to_host(s));
    s->hctl->active = 1;
    UMAG_TRY(push_ctl(s));
    for (int i = 0; i < n; i++) UMAG_TRY(launch_torque(s, 0, 0, nullptr, nullptr, nullptr));
    return UMAG_OK;
}

// engine/energy.go:27-35 GetTotalEnergy and its terms for the current m:
// E[0] total, E[1] demag (engine/demag.go:146), E[2] exchange incl. DMI
// (engine/exchange.go:79), E[3] anisotropy (engine/anisotropy.go:210),
// E[4] Zeeman (engine/zeeman.go:15).  Joules.
// engine/energy.go:36-42 SetTotalEdens: dst = 0, then each term's
// AddDotProduct(dst, prefactor, B_term, M_full) in float32, in the order the
// terms register (anisotropy -1/2 and -1/4, demag -1/2, exchange -1/2,
// Zeeman -1; engine/anisotropy.go:164-190, demag.go:31, exchange.go:34,
// zeeman.go:9)
__global__ void __launch_bounds__(256) k_energy_density(LocalArgs a, const float* __restrict__ vol, float* dst) {
    for (int I = blockIdx.x * blockDim.x + threadIdx.x; I < a.N; I += gridDim.x * blockDim.x) {
        float t[kNE];
        energy_cell_terms(a, vol, I, t);
        float d = 0.0f;
        if (a.anis) {
            d = fa(d, fm(-0.5f, t[2]));
            d = fa(d, fm(-0.25f, t[3]));
        }
        if (a.cubic) {
            d = fa(d, fm(-0.25f, t[5]));
            d = fa(d, fm((float)(-1. / 6.), t[6]));
            d = fa(d, fm(-0.125f, t[7]));
        }
        if (a.bd) d = fa(d, fm(-0.5f, t[0]));
        d = fa(d, fm(-0.5f, t[1]));
        if (a.thermal) d = fa(d, fm(-1.0f, t[8]));
        if (a.zeeman) d = fa(d, fm(-1.0f, t[4]));
        dst[I] = d;
    }
}

int sim_energies(umag_sim* h, double E[5]) {
    SimImpl* s = reinterpret_cast<SimImpl*>(h);
    UMAG_REQUIRE(s && E, "NULL argument");
    if (!s->esum) UMAG_CUDA(cudaMalloc(&s->esum, kNE * sizeof(double)));
    UMAG_TRY(sync_ctl_to_host(s));
    s->hctl->active = 1;
    UMAG_TRY(push_ctl(s));
    if (s->p.enable_demag) {
        PassArgs a = s->pa;
        a.m_sel = 0;
        UMAG_TRY(demag_launch(s->demag, a, S()));
    }
    UMAG_CUDA(cudaMemsetAsync(s->esum, 0, kNE * sizeof(double), S()));
    k_energy_terms<<<grid_for(s->N, 256, 4), 256, 0, S()>>>(s->la, s->p.vol, s->esum);
    UMAG_LAUNCH_CHECK();
    double t[kNE];
    UMAG_CUDA(cudaMemcpyAsync(t, s->esum, sizeof(t), cudaMemcpyDeviceToHost, S()));
    UMAG_CUDA(cudaStreamSynchronize(S()));
    const double V = s->p.cell[0] * s->p.cell[1] * s->p.cell[2];  // engine/energy.go:45-48 cellVolume
    const double Ed = -0.5 * V * t[0], Ee = -0.5 * V * t[1];
    // engine/anisotropy.go:164-206: uniaxial -1/2, -1/4; cubic -1/4, -1/6, -1/8
    const double Ea = V * (-0.5 * t[2] - 0.25 * t[3] - 0.25 * t[5] - t[6] / 6.0 - 0.125 * t[7]);
    const double Ez = -1.0 * V * t[4];
    const double Et = s->la.thermal ? -1.0 * V * t[8] : 0.0;  // engine/temperature.go:124-130
    E[1] = Ed; E[2] = Ee; E[3] = Ea; E[4] = Ez;
    // registration order of the terms (files anisotropy, demag, exchange, temperature, zeeman)
    E[0] = (((Ea + Ed) + Ee) + Et) + Ez;
    return UMAG_OK;
}

// per-cell total energy density (J/m^3) of the current m into dst (device, N floats)
int sim_energy_density(umag_sim* h, float* dst) {
    SimImpl* s = reinterpret_cast<SimImpl*>(h);
    UMAG_REQUIRE(s && dst, "NULL argument");
    UMAG_REQUIRE(!s->batched, "energy density of a batched simulation");
    UMAG_TRY(sync_ctl_to_host(s));
    s->hctl->active = 1;
    UMAG_TRY(push_ctl(s));
    if (s->p.enable_demag) {
        PassArgs a = s->pa;
        a.m_sel = 0;
        UMAG_TRY(demag_launch(s->demag, a, S()));
    }
    k_energy_density<<<grid_for(s->N, 256), 256, 0, S()>>>(s->la, s->p.vol, dst);
    UMAG_LAUNCH_CHECK();
    UMAG_CUDA(cudaStreamSynchronize(S()));
    return UMAG_OK;
}

// switch the stepper / precession (engine/run.go:92-125 SetSolver); the
// stepper restarts (its FSAL torque is recomputed) and the step graphs are rebuilt
static void set_stepper(SimImpl* s, int solver, int precess) {
    if (s->sp.solver != solver || s->la.precess != precess) {
        s->sp.solver = solver;
        s->la.precess = precess;
        drop_graph(s);
    }
    s->need_k1 = true;
}

// engine/relax.go:134-141 relaxSteps: n accepted steps, then time is restored
static int relax_steps(SimImpl* s, int n) {
    UMAG_TRY(sync_ctl_to_host(s));
    const double t0 = s->hctl->t;
    const long long target = s->hctl->nsteps + n;
    s->hctl->stop = INFINITY;
    UMAG_TRY(push_ctl(s));
    s->need_k1 = true;  // runWhile frees the stepper (engine/run.go:207)
    for (int guard = 0; guard < 1000; guard++) {
        UMAG_TRY(sync_ctl_to_host(s));
        if (s->hctl->status != 0)
            return set_error(UMAG_E_SOLVER, "solver failure code %d during relax", s->hctl->status);
        if (s->hctl->nsteps >= target) break;
        UMAG_TRY(run_steps(s, target - s->hctl->nsteps));
    }
    UMAG_TRY(sync_ctl_to_host(s));
    s->hctl->t = t0;
    return push_ctl(s);
}

static int k1_max_norm(SimImpl* s, double* out) {
    UMAG_TRY(sync_ctl_to_host(s));
    const float* k = s->hctl->k[0];
    return max_vec_norm(k, k + s->N, k + 2 * (size_t)s->N, s->N, out);
}
static int k1_dot(SimImpl* s, float* out) {  // opencl.Dot(k1, k1), returned as float32
    UMAG_TRY(sync_ctl_to_host(s));
    double tot = 0;
    for (int c = 0; c < 3; c++) {
        const float* k = s->hctl->k[0] + (size_t)c * s->N;
        double v;
        UMAG_TRY(sum_dot(k, k, s->N, &v));
        tot += v;
    }
    *out = (float)tot;
    return UMAG_OK;
}

// engine/relax.go:23-112 Relax(): RK23 without precession, energy descent in
// chunks of 3 steps, then torque descent with MaxErr lowered by sqrt(2)
// down to 1e-9 (threshold <= 0), or steps while max |torque| > threshold.
int sim_relax(umag_sim* h, double threshold) {
    SimImpl* s = reinterpret_cast<SimImpl*>(h);
    UMAG_REQUIRE(s, "NULL argument");
    UMAG_TRY(sync_ctl_to_host(s));
    const int prev_solver = s->sp.solver, prev_precess = s->la.precess;
    const double prev_err = s->hctl->max_err, prev_fix = s->hctl->fix_dt;
    const int prev_thermal = s->la.thermal;
    set_stepper(s, 3, 0);
    s->la.thermal = 0;  // engine/effectivefield.go:20: no B_therm while relaxing
    if (prev_thermal) drop_graph(s);  // the captured steps bake the flag in
    s->hctl->fix_dt = 0;
    UMAG_TRY(push_ctl(s));
    auto body = [&]() -> int {
        const int n = 3;  // evaluate the energy every 3 steps (relax.go:54)
        double E[5];
        UMAG_TRY(relax_steps(s, n));
        UMAG_TRY(sim_energies(h, E));
        double E0 = E[0];
        UMAG_TRY(relax_steps(s, n));
        UMAG_TRY(sim_energies(h, E));
        double E1 = E[0];
        for (int guard = 0; E1 < E0 && guard < 1000000; guard++) {
            UMAG_TRY(relax_steps(s, n));
            UMAG_TRY(sim_energies(h, E));
            E0 = E1;
            E1 = E[0];
        }
        if (threshold > 0) {
            for (;;) {
                double mt;
                UMAG_TRY(k1_max_norm(s, &mt));
                for (int guard = 0; mt > threshold && guard < 1000000; guard++) {
                    UMAG_TRY(relax_steps(s, n));
                    UMAG_TRY(k1_max_norm(s, &mt));
                }
                UMAG_TRY(sync_ctl_to_host(s));
                s->hctl->max_err /= std::sqrt(2.0);
                UMAG_TRY(push_ctl(s));
                if (s->hctl->max_err < 1e-9) break;
            }
        } else {
            float T0 = 0, T1;
            UMAG_TRY(k1_dot(s, &T1));
            for (;;) {
                UMAG_TRY(sync_ctl_to_host(s));
                if (!(s->hctl->max_err > 1e-9)) break;
                s->hctl->max_err /= std::sqrt(2.0);
                UMAG_TRY(push_ctl(s));
                UMAG_TRY(relax_steps(s, n));
                T0 = T1;
                UMAG_TRY(k1_dot(s, &T1));
                for (int guard = 0; T1 < T0 && guard < 1000000; guard++) {
                    UMAG_TRY(relax_steps(s, n));
                    T0 = T1;
                    UMAG_TRY(k1_dot(s, &T1));
                }
            }
        }
        return UMAG_OK;
    };
    const int st = body();
    // restore the caller's settings (relax.go:36-45)
    sync_ctl_to_host(s);
    s->hctl->max_err = prev_err;
    s->hctl->fix_dt = prev_fix;
    push_ctl(s);
    s->la.thermal = prev_thermal;
    drop_graph(s);
    set_stepper(s, prev_solver, prev_precess);
    return st;
}

// Reassigning solver settings between runs: SetSolver (engine/run.go:92-125,
// the stepper restarts), FixDt, MaxErr, RelErr, MinDt, MaxDt, Headroom,
// MinSlope, GammaLL.  The current time and dt are kept (assigning FixDt = 0
// resumes adaptive stepping from the last dt, as adaptDt does).
int sim_set_solver(umag_sim* h, const umag_solver_params* sp) {
    SimImpl* s = reinterpret_cast<SimImpl*>(h);
    UMAG_REQUIRE(s && sp, "NULL argument");
    UMAG_REQUIRE(!s->batched, "solver settings of a batched simulation");
    UMAG_REQUIRE(sp->solver >= 1 && sp->solver <= 5,
                 "solver must be 1 (Euler), 2 (Heun), 3 (RK23), 4 (RK4) or 5 (RK45DP)");
    UMAG_TRY(sync_ctl_to_host(s));
    DevCtl& c = *s->hctl;
    c.max_err = sp->max_err; c.rel_err = sp->rel_err; c.min_dt = sp->min_dt; c.max_dt = sp->max_dt;
    c.fix_dt = sp->fix_dt; c.headroom = sp->headroom; c.min_slope = sp->min_slope;
    if (c.therm_gv != 0) c.therm_gv = sp->gamma_ll * (s->p.cell[0] * s->p.cell[1] * s->p.cell[2]);
    c.gamma = sp->gamma_ll;
    UMAG_TRY(push_ctl(s));
    const double dt_keep = s->sp.dt;
    const int prev = s->sp.solver;
    s->sp = *sp;
    s->sp.dt = dt_keep;
    s->sp.solver = prev;
    set_stepper(s, sp->solver, s->la.precess);  // new graphs only when the stepper changes
    return UMAG_OK;
}

// Launch shapes of the per-cell kernels: any valid shape gives the same
// results (per-cell arithmetic, max reductions), only the speed differs.
int sim_get_tuning(umag_sim* h, umag_tuning* t) {
    SimImpl* s = reinterpret_cast<SimImpl*>(h);
    UMAG_REQUIRE(s && t, "NULL argument");
    *t = s->tune;
    return UMAG_OK;
}
int sim_set_tuning(umag_sim* h, const umag_tuning* t) {
    SimImpl* s = reinterpret_cast<SimImpl*>(h);
    UMAG_REQUIRE(s && t, "NULL argument");
    const int bx = t->torque_block[0], by = t->torque_block[1];
    UMAG_REQUIRE(bx >= 32 && bx % 32 == 0 && by >= 1 && bx * by <= 256, "torque block %dx%d", bx, by);
    UMAG_REQUIRE(t->stage_threads == 64 || t->stage_threads == 128 || t->stage_threads == 256,
                 "stage threads %d", t->stage_threads);
    UMAG_REQUIRE(t->stage_waves >= 1 && t->stage_waves <= 64 && t->err_waves >= 1 && t->err_waves <= 64,
                 "waves must be 1..64");
    UMAG_REQUIRE(t->torque_tma == 0 || t->torque_tma == 1, "torque_tma must be 0 or 1");
    UMAG_CUDA(cudaStreamSynchronize(S()));
    s->tune = *t;
    if (!s->batched) tile_setup(s);  // the box follows the block shape
    drop_graph(s);  // the captured launches carry the old shapes
    return UMAG_OK;
}

// Reassigning a material parameter between runs (engine/parameter.go
// setRegion / SetValue): a per-cell device map (the caller keeps it alive
// while the simulation uses it) or NULL with a uniform value.
int sim_set_param(umag_sim* h, int which, const float* values, float mul) {
    SimImpl* s = reinterpret_cast<SimImpl*>(h);
    UMAG_REQUIRE(s, "NULL argument");
    UMAG_REQUIRE(!s->batched, "parameters of a batched simulation");
    umag_sim_params& p = s->p;
    switch (which) {
    case UMAG_PARAM_MSAT: p.Ms = values; p.Ms_mul = mul; break;
    case UMAG_PARAM_ALPHA: p.alpha = values; p.alpha_mul = mul; break;
    case UMAG_PARAM_KU1: p.Ku1 = values; p.Ku1_mul = mul; break;
    case UMAG_PARAM_KU2: p.Ku2 = values; p.Ku2_mul = mul; break;
    case UMAG_PARAM_TEMP: p.temp = values; p.temp_mul = mul; break;
    case UMAG_PARAM_KC1: p.Kc1 = values; p.Kc1_mul = mul; break;
    case UMAG_PARAM_KC2: p.Kc2 = values; p.Kc2_mul = mul; break;
    case UMAG_PARAM_KC3: p.Kc3 = values; p.Kc3_mul = mul; break;
    default:
        if (which >= UMAG_PARAM_ANISU_X && which <= UMAG_PARAM_ANISU_X + 2) {
            p.anisU[which - UMAG_PARAM_ANISU_X] = values;
            p.anisU_mul[which - UMAG_PARAM_ANISU_X] = mul;
        } else if (which >= UMAG_PARAM_ANISC1_X && which <= UMAG_PARAM_ANISC1_X + 2) {
            p.anisC1[which - UMAG_PARAM_ANISC1_X] = values;
            p.anisC1_mul[which - UMAG_PARAM_ANISC1_X] = mul;
        } else if (which >= UMAG_PARAM_ANISC2_X && which <= UMAG_PARAM_ANISC2_X + 2) {
            p.anisC2[which - UMAG_PARAM_ANISC2_X] = values;
            p.anisC2_mul[which - UMAG_PARAM_ANISC2_X] = mul;
        } else {
            return set_error(UMAG_E_ARG, "unknown parameter %d", which);
        }
    }
    UMAG_CUDA(cudaStreamSynchronize(S()));
    drop_graph(s);  // the captured launches bake the old arguments in
    UMAG_TRY(local_from_params(s));
    if (which == UMAG_PARAM_TEMP) {  // engine/temperature.go:111: gamma V of the noise amplitude
        UMAG_TRY(sync_ctl_to_host(s));
        DevCtl& c = *s->hctl;
        c.therm_gv = s->la.thermal ? s->sp.gamma_ll * (p.cell[0] * p.cell[1] * p.cell[2]) : 0.0;
        if (c.therm_gv != 0) c.k2 = (float)(2 * kBoltzmann / (c.therm_gv * c.dt));
        UMAG_TRY(push_ctl(s));
    }
    s->need_k1 = true;  // the FSAL torque belongs to the old parameters
    return UMAG_OK;
}

// ================================================================ ensembles
// Many independent simulations advanced together (no reference counterpart:
// uMagNUS runs one simulation per process).  Instances with the same mesh
// form a class, run as one batched SimImpl: every field / stage / error
// kernel handles all instances of the class in one launch (grid extended by
// the instance index) and one controller thread per instance keeps its own
// time, dt and accept/reject decisions.  One CUDA graph steps every class,
// the classes on parallel branches.
//
// Scheduling: each class has its own stream and its own graph of
// graph_steps steps; the host keeps every unfinished class's stream fed with
// chunks of replays and polls each class on its own (an event after the
// chunk and its state copy), so a cheap class never waits for an expensive
// one.  When a chunk leaves at most 3/4 of a class's batch still running,
// the running instances are compacted to the front of the batch (their
// controller records, parameters and per-instance indices permuted; the
// state buffers stay where they are, the records point at them) and the
// class's graph is recaptured for the smaller batch, so finished instances
// stop costing launches.  Every instance's arithmetic is unchanged.
constexpr int kEnsUnit = 4;        // steps of one graph of a class
constexpr int kEnsReplay = 16;     // steps that `chunk` and `max_replays` count in
constexpr size_t kEnsGraphs = 12;  // graphs a class keeps
constexpr int kEnsCompact = 64;    // steps that must be left for a new batch size to pay
struct EnsClass {
    SimImpl* s = nullptr;
    // a general instance: one simulation made by sim_new from a full
    // umag_sim_params (region maps, per-cell maps, geometry, PBC, every
    // term), stepped by the single-simulation kernels on the class's stream
    bool general = false;
    std::vector<int> members;  // ensemble index of each batch slot
    float2* spec = nullptr;    // nb spectrum scratch copies
    float* params = nullptr;   // device: Ms[n_all], A00[n_all], D00[n_all]
    std::vector<float> hparams;  // host copy of params (permuted with the slots)
    int n_all = 0;             // instances of the class; the first s->nb slots are in the batch
    cudaStream_t st = nullptr;
    cudaEvent_t done = nullptr;
    std::map<int, cudaGraphExec_t> graphs;  // kEnsUnit steps, by batch size
    bool busy = false, finished = false;
    long long units = 0;  // queued in this run
};
struct EnsImpl {
    std::vector<EnsClass> cls;
    std::vector<std::pair<int, int>> where;  // instance -> (class, slot in class)
    umag_solver_params sp;
};

static void ens_drop_graphs(EnsClass& c) {
    for (auto& g : c.graphs) cudaGraphExecDestroy(g.second);
    c.graphs.clear();
}
static void ens_class_free(EnsClass& c) {
    ens_drop_graphs(c);
    if (c.s && c.general) {
        sim_free(reinterpret_cast<umag_sim*>(c.s));
        c.s = nullptr;
    }
    if (c.s) {
        SimImpl* s = c.s;
        drop_graph(s);
        if (s->demag) demag_free(s->demag);
        cudaFree(s->bufs);
        cudaFree(s->bd);
        cudaFree(s->zero_regions);
        cudaFree(s->kc_dev);
        cudaFree(s->ip_dev);
        cudaFree(s->ctl);
        if (s->hctl) cudaFreeHost(s->hctl);
        delete s;
        c.s = nullptr;
    }
    cudaFree(c.spec);
    cudaFree(c.params);
    if (c.st) cudaStreamDestroy(c.st);
    if (c.done) cudaEventDestroy(c.done);
    c.spec = nullptr;
    c.params = nullptr;
    c.st = nullptr;
    c.done = nullptr;
}

int ens_free(umag_ens* h) {
    EnsImpl* e = reinterpret_cast<EnsImpl*>(h);
    if (!e) return UMAG_OK;
    cudaDeviceSynchronize();
    for (auto& c : e->cls) ens_class_free(c);
    delete e;
    return UMAG_OK;
}

// one class: nb instances of mesh N, cell, with the listed parameters
static int ens_class_new(EnsClass& C, const umag_ens_instance* in, const std::vector<int>& members,
                         const umag_solver_params* sp, int demag) {
    const int nb = (int)members.size();
    const umag_ens_instance& r0 = in[members[0]];
    SimImpl* s = new SimImpl();
    C.s = s;
    C.members = members;
    C.n_all = nb;
    s->nb = nb;
    s->batched = true;
    s->sp = *sp;
    memset(&s->p, 0, sizeof(s->p));
    for (int i = 0; i < 3; i++) { s->p.N[i] = r0.N[i]; s->p.cell[i] = r0.cell[i]; }
    s->p.enable_demag = demag;
    s->p.precess = 1;
    s->N = r0.N[0] * r0.N[1] * r0.N[2];
    s->g = Mesh3{r0.N[0], r0.N[1], r0.N[2], 0};
    const size_t n3 = 3 * (size_t)s->N;
    UMAG_CUDA(cudaStreamCreateWithFlags(&C.st, cudaStreamNonBlocking));
    UMAG_CUDA(cudaEventCreateWithFlags(&C.done, cudaEventDisableTiming));
    UMAG_CUDA(cudaMalloc(&s->bufs, sizeof(float) * n3 * 10 * nb));
    UMAG_CUDA(cudaMemsetAsync(s->bufs, 0, sizeof(float) * n3 * 10 * nb, S()));
    UMAG_CUDA(cudaMalloc(&s->zero_regions, s->N));
    UMAG_CUDA(cudaMemsetAsync(s->zero_regions, 0, s->N, S()));
    s->p.regions = s->zero_regions;
    if (demag) {
        int pbc[3] = {0, 0, 0};
        UMAG_TRY(demag_new_newell(r0.N[0], r0.N[1], r0.N[2], pbc, r0.cell[0], r0.cell[1], r0.cell[2], 32, 0, &s->demag));
        UMAG_CUDA(cudaMalloc(&s->bd, sizeof(float) * n3 * nb));
        UMAG_CUDA(cudaMemsetAsync(s->bd, 0, sizeof(float) * n3 * nb, S()));
    }
    UMAG_CUDA(cudaMalloc(&s->ctl, sizeof(DevCtl) * nb));
    UMAG_CUDA(cudaMallocHost(&s->hctl, sizeof(DevCtl) * nb));
    memset(s->hctl, 0, sizeof(DevCtl) * nb);
    for (int b = 0; b < nb; b++) {
        DevCtl& c = s->hctl[b];
        float* base = s->bufs + (size_t)b * 10 * n3;
        c.m = base;
        for (int i = 0; i < 2; i++) c.mw[i] = base + (1 + i) * n3;
        for (int i = 0; i < 7; i++) c.k[i] = base + (3 + i) * n3;
        c.bd = s->bd ? s->bd + (size_t)b * n3 : nullptr;
        c.dt = sp->dt;
        c.stop = INFINITY;
        c.max_err = sp->max_err; c.rel_err = sp->rel_err; c.min_dt = sp->min_dt; c.max_dt = sp->max_dt;
        c.fix_dt = sp->fix_dt; c.headroom = sp->headroom; c.min_slope = sp->min_slope; c.gamma = sp->gamma_ll;
        c.active = 1;
    }
    UMAG_TRY(push_ctl(s));
    // per-instance uniform values: Ms, and the region-(0,0) LUT entries the
    // plain engine would use (engine/exchange.go:193-201 harmonic mean, float32)
    std::vector<float> hp(3 * nb);
    bool dmi = false, anis = false, zee = false;
    for (int b = 0; b < nb; b++) {
        const umag_ens_instance& r = in[members[b]];
        hp[b] = r.Ms;
        hp[nb + b] = 2.0f / (1.0f / r.Aex + 1.0f / r.Aex);
        const float D = r.Dind;
        hp[2 * nb + b] = D == 0.0f ? 0.0f : 2.0f / (1.0f / D + 1.0f / D);
        dmi |= D != 0.0f;
        anis |= r.Ku1 != 0.0f || r.Ku2 != 0.0f;
        zee |= r.B_ext[0] != 0.0f || r.B_ext[1] != 0.0f || r.B_ext[2] != 0.0f;
    }
    UMAG_CUDA(cudaMalloc(&C.params, sizeof(float) * 3 * nb));
    UMAG_CUDA(cudaMemcpyAsync(C.params, hp.data(), sizeof(float) * 3 * nb, cudaMemcpyHostToDevice, S()));
    C.hparams = hp;
    UMAG_CUDA(cudaStreamSynchronize(S()));
    UMAG_CUDA(cudaMalloc(&s->ip_dev, sizeof(InstParams) * nb));
    LocalArgs& la = s->la;
    la.g = s->g;
    la.N = s->N;
    la.ctl = s->ctl;
    la.bd = nullptr;
    la.regions = s->zero_regions;
    la.cx = (float)r0.cell[0]; la.cy = (float)r0.cell[1]; la.cz = (float)r0.cell[2];
    la.wx = (float)(2 / (r0.cell[0] * r0.cell[0]));
    la.wy = (float)(2 / (r0.cell[1] * r0.cell[1]));
    la.wz = (float)(2 / (r0.cell[2] * r0.cell[2]));
    la.dmi = dmi;
    la.openbc = 0;
    la.anis = anis;
    la.zeeman = zee;
    la.precess = 1;
    la.ms_uniform = 1; la.alpha_uniform = 1; la.anis_uniform = 1;
    la.ip = s->ip_dev;
    std::vector<InstParams> hip(nb);
    for (int b = 0; b < nb; b++) {  // uniform constants of each instance, bit-identical to the plain engine's
        const umag_ens_instance& r = in[members[b]];
        LocalArgs t = la;
        t.aLUT = C.params + nb + b;
        t.dLUT = C.params + 2 * nb + b;
        t.alpha_mul = r.alpha;
        t.Ms_mul = r.Ms;
        t.up = UniaxParams{nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, r.Ms, r.Ku1, r.Ku2,
                           r.anisU[0], r.anisU[1], r.anisU[2]};
        k_local_consts<<<1, 1, 0, S()>>>(t, &s->ip_dev[b].kc);
        UMAG_LAUNCH_CHECK();
        hip[b].alpha_mul = r.alpha;
        hip[b].Ms_mul = r.Ms;
        hip[b].dmi = r.Dind != 0.0f;
        for (int c = 0; c < 3; c++) hip[b].bext[c] = r.B_ext[c];
    }
    UMAG_CUDA(cudaStreamSynchronize(S()));
    // fill the non-kc fields without touching kc
    for (int b = 0; b < nb; b++)
        UMAG_CUDA(cudaMemcpyAsync(reinterpret_cast<char*>(s->ip_dev + b) + offsetof(InstParams, alpha_mul),
                                  reinterpret_cast<char*>(&hip[b]) + offsetof(InstParams, alpha_mul),
                                  sizeof(InstParams) - offsetof(InstParams, alpha_mul), cudaMemcpyHostToDevice, S()));
    UMAG_CUDA(cudaStreamSynchronize(S()));
    if (demag) {
        fill_pass_args(s->demag, s->pa);
        const long spec_elems = 3L * s->demag->F[2] * s->demag->N[1] * s->demag->Lx;  // one plan's spectrum
        UMAG_CUDA(cudaMalloc(&C.spec, sizeof(float2) * spec_elems * nb));
        UMAG_CUDA(cudaMemsetAsync(C.spec, 0, sizeof(float2) * spec_elems * nb, S()));
        s->pa.spec = C.spec;
        s->pa.spec_stride = spec_elems;
        s->pa.m_ind = &s->ctl[0].m;
        s->pa.m_ind_w = &s->ctl[0].mw[0];
        s->pa.active = &s->ctl[0].active;
        s->pa.fault = &s->ctl[0].status;
        s->pa.ctl_stride = sizeof(DevCtl);
        s->pa.vol = nullptr;
        s->pa.Ms = nullptr;
        s->pa.Ms_mul = 0.0f;
        s->pa.ms_mul_b = C.params;
        s->pa.ncell = s->N;
        for (int c = 0; c < 3; c++) s->pa.B[c] = s->bd + (size_t)c * s->N;
        s->pa.b_stride = (long)n3;
    }
    return UMAG_OK;
}

// a class of one general instance: the simulation sim_new makes from the
// full parameter record, with its own stream and completion event
static int ens_class_new_general(EnsClass& C, int member, const umag_sim_params* p, const umag_solver_params* sp) {
    C.general = true;
    C.members = {member};
    C.n_all = 1;
    umag_sim* h = nullptr;
    UMAG_TRY(sim_new(p, sp, &h));
    C.s = reinterpret_cast<SimImpl*>(h);
    UMAG_CUDA(cudaStreamCreateWithFlags(&C.st, cudaStreamNonBlocking));
    UMAG_CUDA(cudaEventCreateWithFlags(&C.done, cudaEventDisableTiming));
    return UMAG_OK;
}

int ens_new(int n, const umag_ens_instance* in, const umag_solver_params* sp, int demag, umag_ens** out) {
    return ens_new_general(n, in, nullptr, sp, demag, out);
}

int ens_new_general(int n, const umag_ens_instance* in, const umag_sim_params* const* general,
                    const umag_solver_params* sp, int demag, umag_ens** out) {
    UMAG_TRY(ensure_init());
    UMAG_REQUIRE(n > 0 && sp && out, "bad argument");
    UMAG_REQUIRE(sp->solver >= 1 && sp->solver <= 5, "unknown solver");
    for (int i = 0; i < n; i++)
        UMAG_REQUIRE(in || (general && general[i]), "instance %d: no uniform record and no general parameters", i);
    EnsImpl* e = new EnsImpl();
    e->sp = *sp;
    e->where.resize(n);
    auto fail = [&](int code) { ens_free(reinterpret_cast<umag_ens*>(e)); return code; };
    // classes: same mesh and cell size; each general instance is a class of its own
    std::vector<std::vector<int>> groups;
    std::vector<int> gen_of;  // class -> general instance, or -1
    for (int i = 0; i < n; i++) {
        if (general && general[i]) {
            e->where[i] = {(int)groups.size(), 0};
            groups.push_back({i});
            gen_of.push_back(i);
            continue;
        }
        const umag_ens_instance& r = in[i];
        if (r.N[0] <= 0 || r.N[1] <= 0 || r.N[2] <= 0) return fail(set_error(UMAG_E_ARG, "instance %d: bad mesh", i));
        if (!(r.Ms > 0) || !(r.Aex > 0)) return fail(set_error(UMAG_E_ARG, "instance %d: Ms and Aex must be > 0", i));
        int g = -1;
        for (size_t k = 0; k < groups.size(); k++) {
            if (gen_of[k] >= 0) continue;
            const umag_ens_instance& q = in[groups[k][0]];
            if (q.N[0] == r.N[0] && q.N[1] == r.N[1] && q.N[2] == r.N[2] && q.cell[0] == r.cell[0] &&
                q.cell[1] == r.cell[1] && q.cell[2] == r.cell[2])
                g = (int)k;
        }
        if (g < 0) { groups.push_back({}); gen_of.push_back(-1); g = (int)groups.size() - 1; }
        e->where[i] = {g, (int)groups[g].size()};
        groups[g].push_back(i);
    }
    e->cls.resize(groups.size());
    for (size_t k = 0; k < groups.size(); k++) {
        const int st = gen_of[k] >= 0 ? ens_class_new_general(e->cls[k], gen_of[k], general[gen_of[k]], sp)
                                      : ens_class_new(e->cls[k], in, groups[k], sp, demag);
        if (st != UMAG_OK) return fail(st);
    }
    *out = reinterpret_cast<umag_ens*>(e);
    return UMAG_OK;
}

// every slot's controller record to the host (the batch may be smaller
// than the class after compaction; records past it do not change)
static int ens_sync_all(EnsClass& C) {
    SimImpl* s = C.s;
    UMAG_CUDA(cudaMemcpyAsync(s->hctl, s->ctl, sizeof(DevCtl) * C.n_all, cudaMemcpyDeviceToHost, S()));
    UMAG_CUDA(cudaStreamSynchronize(S()));
    return UMAG_OK;
}
static int ens_push_all(EnsClass& C) {
    SimImpl* s = C.s;
    UMAG_CUDA(cudaMemcpyAsync(s->ctl, s->hctl, sizeof(DevCtl) * C.n_all, cudaMemcpyHostToDevice, S()));
    UMAG_CUDA(cudaStreamSynchronize(S()));
    return UMAG_OK;
}

static SimImpl* ens_sim(EnsImpl* e, int i, int* b) {
    const auto& w = e->where[i];
    *b = w.second;
    return e->cls[w.first].s;
}

int ens_set_m(umag_ens* h, int i, const float* host_m) {
    EnsImpl* e = reinterpret_cast<EnsImpl*>(h);
    UMAG_REQUIRE(e && host_m && i >= 0 && i < (int)e->where.size(), "bad argument");
    int b;
    SimImpl* s = ens_sim(e, i, &b);
    UMAG_TRY(ens_sync_all(e->cls[e->where[i].first]));
    float* m = s->hctl[b].m;
    // on the library stream, so that the normalisation below sees the copy
    UMAG_CUDA(cudaMemcpyAsync(m, host_m, sizeof(float) * 3 * s->N, cudaMemcpyHostToDevice, S()));
    // engine/magnetization.go:34 (the geometry mask of a general instance; none in a batch)
    UMAG_TRY(normalize(m, m + s->N, m + 2 * (size_t)s->N, s->p.vol, s->N));
    UMAG_CUDA(cudaDeviceSynchronize());
    s->need_k1 = true;
    return UMAG_OK;
}

int ens_get_m(umag_ens* h, int i, float* host_m) {
    EnsImpl* e = reinterpret_cast<EnsImpl*>(h);
    UMAG_REQUIRE(e && host_m && i >= 0 && i < (int)e->where.size(), "bad argument");
    int b;
    SimImpl* s = ens_sim(e, i, &b);
    UMAG_TRY(ens_sync_all(e->cls[e->where[i].first]));
    UMAG_CUDA(cudaMemcpyAsync(host_m, s->hctl[b].m, sizeof(float) * 3 * s->N, cudaMemcpyDeviceToHost, S()));
    UMAG_CUDA(cudaStreamSynchronize(S()));
    return UMAG_OK;
}

int ens_get_state(umag_ens* h, int i, umag_solver_state* st) {
    EnsImpl* e = reinterpret_cast<EnsImpl*>(h);
    UMAG_REQUIRE(e && st && i >= 0 && i < (int)e->where.size(), "bad argument");
    int b;
    SimImpl* s = ens_sim(e, i, &b);
    UMAG_TRY(ens_sync_all(e->cls[e->where[i].first]));
    const DevCtl& c = s->hctl[b];
    st->time = c.t; st->dt = c.dt; st->last_err = c.last_err; st->peak_err = c.peak_err;
    st->last_torque = c.last_torque; st->nsteps = c.nsteps; st->nundone = c.nundone; st->nevals = c.nevals;
    st->status = c.status;
    return UMAG_OK;
}

// kEnsUnit steps of class C's current batch, captured on its stream (which is
// idle).  A batch size comes back in every run, so its graph is kept.
static int ens_capture(EnsClass& C) {
    if (C.graphs.count(C.s->nb)) return UMAG_OK;
    if (C.graphs.size() >= kEnsGraphs) ens_drop_graphs(C);
    cudaGraphExec_t g = nullptr;
    g_launch_stream = C.st;
    const int st = capture_steps(C.s, kEnsUnit, &g);
    g_launch_stream = nullptr;
    if (st == UMAG_OK) C.graphs[C.s->nb] = g;
    return st;
}

// Compact the running instances of class C to the front of its batch (the
// host records are fresh: its stream is idle).  Slot k takes the instance of
// old slot order[k]: its controller record (which points at its own state
// buffers; the demag-field scratch pointer is the slot's), its parameters
// and its uniform constants.
static int ens_compact(EnsImpl* e, int ci) {
    EnsClass& C = e->cls[ci];
    if (C.general) return UMAG_OK;  // one instance: nothing to compact
    SimImpl* s = C.s;
    const int nb = s->nb;
    std::vector<int> order;
    for (int b = 0; b < nb; b++)
        if (s->hctl[b].t < s->hctl[b].stop && s->hctl[b].status == 0) order.push_back(b);
    const int na = (int)order.size();
    if (na == 0 || 4 * na > 3 * nb) return UMAG_OK;
    // A smaller batch needs a graph of its own, about a millisecond of this
    // thread for 100 launches; what a finished instance costs is the early exit
    // of its CTAs.  (48 films of up to 134 steps: 34.9 ms
    // compacting at every poll, 21.6 ms without.)
    long long left = 0;
    for (int b = 0; b < nb; b++) left = std::max(left, steps_left(s->hctl[b]));
    if (left < kEnsCompact && !C.graphs.count(na)) return UMAG_OK;
    for (int b = 0; b < nb; b++)
        if (!(s->hctl[b].t < s->hctl[b].stop && s->hctl[b].status == 0)) order.push_back(b);
    std::vector<DevCtl> ctl(nb);
    std::vector<int> mem(nb);
    std::vector<float> hp = C.hparams;
    const size_t n3 = 3 * (size_t)s->N;
    InstParams* tmp = nullptr;
    UMAG_CUDA(cudaMalloc(&tmp, sizeof(InstParams) * nb));
    for (int k = 0; k < nb; k++) {
        const int o = order[k];
        ctl[k] = s->hctl[o];
        if (s->bd) ctl[k].bd = s->bd + (size_t)k * n3;
        mem[k] = C.members[o];
        for (int q = 0; q < 3; q++) hp[q * C.n_all + k] = C.hparams[q * C.n_all + o];
        UMAG_CUDA(cudaMemcpyAsync(tmp + k, s->ip_dev + o, sizeof(InstParams), cudaMemcpyDeviceToDevice, S()));
    }
    UMAG_CUDA(cudaMemcpyAsync(s->ip_dev, tmp, sizeof(InstParams) * nb, cudaMemcpyDeviceToDevice, S()));
    UMAG_CUDA(cudaStreamSynchronize(S()));
    cudaFree(tmp);
    for (int k = 0; k < nb; k++) {
        s->hctl[k] = ctl[k];
        C.members[k] = mem[k];
        e->where[mem[k]] = {ci, k};
    }
    C.hparams = hp;
    UMAG_CUDA(cudaMemcpyAsync(C.params, hp.data(), sizeof(float) * hp.size(), cudaMemcpyHostToDevice, S()));
    UMAG_TRY(ens_push_all(C));
    s->nb = na;
    return ens_capture(C);
}

// engine/run.go:190 Run(seconds) for every instance: each runs until its own
// time reaches start + seconds (its dt honours that alarm).  Classes advance
// independently, at most `chunk` * kEnsReplay steps at a time (and max_replays *
// kEnsReplay in all).  A block covers three quarters of what its slowest instance
// needs by its last time step (first 8 steps, while the time step still
// grows): steps past the stop time do nothing but cost their launches.
int ens_run(umag_ens* h, double seconds, int chunk, long long max_replays) {
    EnsImpl* e = reinterpret_cast<EnsImpl*>(h);
    UMAG_REQUIRE(e && seconds >= 0, "bad argument");
    if (chunk <= 0) chunk = 8;
    const long long per = kEnsReplay / kEnsUnit, max_units = max_replays > (1LL << 60) ? 1LL << 62 : max_replays * per;
    for (auto& C : e->cls) {
        SimImpl* s = C.s;
        UMAG_TRY(ens_sync_all(C));
        s->nb = C.n_all;  // every instance takes part again
        for (int b = 0; b < s->nb; b++) {
            s->hctl[b].stop = s->hctl[b].t + seconds;
            s->hctl[b].alarm = s->hctl[b].stop;
        }
        UMAG_TRY(ens_push_all(C));
        s->need_k1 = true;  // RunWhile frees the stepper (engine/run.go:207)
        UMAG_TRY(ensure_k1(s));
        UMAG_TRY(ens_capture(C));
        C.busy = false;
        C.finished = false;
        C.units = 0;
    }
    UMAG_CUDA(cudaDeviceSynchronize());
    for (;;) {
        bool all_done = true, progressed = false;
        for (size_t ci = 0; ci < e->cls.size(); ci++) {
            EnsClass& C = e->cls[ci];
            SimImpl* s = C.s;
            if (C.finished) continue;
            all_done = false;
            if (C.busy) {
                const cudaError_t q = cudaEventQuery(C.done);
                if (q == cudaErrorNotReady) continue;
                if (q != cudaSuccess) return set_error(UMAG_E_CUDA, "ensemble class %zu: %s", ci, cudaGetErrorString(q));
                C.busy = false;
                progressed = true;
                int running = 0;
                for (int b = 0; b < s->nb; b++) {
                    const DevCtl& d = s->hctl[b];
                    if (d.status != 0)
                        return set_error(UMAG_E_SOLVER, "instance %d: solver failure code %d at t=%g", C.members[b],
                                         d.status, d.t);
                    running += d.t < d.stop;
                }
                if (running == 0 || C.units >= max_units) {
                    C.finished = true;
                    continue;
                }
                UMAG_TRY(ens_compact(e, (int)ci));
            }
            // the next block, then the batch's records back to the host
            long long last = 0;
            for (int b = 0; b < s->nb; b++) last = std::max(last, steps_left(s->hctl[b]));
            const long long steps = C.units == 0 ? 8 : std::max((3 * last + 3) / 4, std::min(last, 8LL));
            const long long want = (steps + kEnsUnit - 1) / kEnsUnit;
            for (long long k = std::min(want, chunk * per); k > 0 && C.units < max_units; k--, C.units++)
                UMAG_CUDA(cudaGraphLaunch(C.graphs[s->nb], C.st));
            UMAG_CUDA(cudaMemcpyAsync(s->hctl, s->ctl, sizeof(DevCtl) * s->nb, cudaMemcpyDeviceToHost, C.st));
            UMAG_CUDA(cudaEventRecord(C.done, C.st));
            C.busy = true;
            progressed = true;
        }
        if (all_done) break;
        if (!progressed) std::this_thread::yield();
    }
    UMAG_CUDA(cudaDeviceSynchronize());
    return UMAG_OK;
}

int ens_count(umag_ens* h, int* n_instances, int* n_classes) {
    EnsImpl* e = reinterpret_cast<EnsImpl*>(h);
    UMAG_REQUIRE(e, "NULL argument");
    if (n_instances) *n_instances = (int)e->where.size();
    if (n_classes) *n_classes = (int)e->cls.size();
    return UMAG_OK;
}

int ens_class_info(umag_ens* h, int cls, int N[3], int* n_instances) {
    EnsImpl* e = reinterpret_cast<EnsImpl*>(h);
    UMAG_REQUIRE(e && N && n_instances, "NULL argument");
    UMAG_REQUIRE(cls >= 0 && cls < (int)e->cls.size(), "class %d out of range", cls);
    const SimImpl* s = e->cls[cls].s;
    for (int i = 0; i < 3; i++) N[i] = s->p.N[i];
    *n_instances = e->cls[cls].n_all;
    return UMAG_OK;
}

int ens_class_general(umag_ens* h, int cls, int* general) {
    EnsImpl* e = reinterpret_cast<EnsImpl*>(h);
    UMAG_REQUIRE(e && general, "NULL argument");
    UMAG_REQUIRE(cls >= 0 && cls < (int)e->cls.size(), "class %d out of range", cls);
    *general = e->cls[cls].general ? 1 : 0;
    return UMAG_OK;
}

int ens_get_tuning(umag_ens* h, int cls, umag_tuning* t) {
    EnsImpl* e = reinterpret_cast<EnsImpl*>(h);
    UMAG_REQUIRE(e && t, "NULL argument");
    UMAG_REQUIRE(cls >= 0 && cls < (int)e->cls.size(), "class %d out of range", cls);
    *t = e->cls[cls].s->tune;
    return UMAG_OK;
}

// the class's launches take the new shapes at its next capture
int ens_set_tuning(umag_ens* h, int cls, const umag_tuning* t) {
    EnsImpl* e = reinterpret_cast<EnsImpl*>(h);
    UMAG_REQUIRE(e && t, "NULL argument");
    UMAG_REQUIRE(cls >= 0 && cls < (int)e->cls.size(), "class %d out of range", cls);
    EnsClass& C = e->cls[cls];
    UMAG_TRY(sim_set_tuning(reinterpret_cast<umag_sim*>(C.s), t));
    ens_drop_graphs(C);
    return UMAG_OK;
}

int sim_launches_per_step(umag_sim* h, int* n) {
    SimImpl* s = reinterpret_cast<SimImpl*>(h);
    UMAG_REQUIRE(s && n, "NULL argument");
    *n = s->launches_per_step;
    return UMAG_OK;
}

}  // namespace umag
