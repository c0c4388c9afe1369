// demag.cuh -- demag plan shared by the device-op API and the engine.
#pragma once
#include <vector>

#include <cuda.h>

#include "common.cuh"
#include "fft.cuh"

constexpr int kPassThreads = 256;   // passes A and C
constexpr int kPassBThreads = 512;  // pass B
constexpr int kChunkW = 32;         // kx columns per z-transform block in passes A/C

namespace umag {
struct PassArgs;
// the kernels of one plan on line transforms (demag_lines.cuh) and, where
// a mesh has them, the fused x/z passes (demag_fast.cu).  The instance of a
// batched launch is blockIdx.z (fused passes: kernels of their own).
struct Passes {
    void (*xf)(PassArgs) = nullptr;
    void (*xi)(PassArgs) = nullptr;
    void (*zf)(PassArgs) = nullptr;  // NULL: one layer
    void (*zi)(PassArgs) = nullptr;
    void (*y)(PassArgs) = nullptr;
    size_t smem_x = 0, smem_y3 = 0, smem_y2 = 0;  // y: of 3D plans and of one layer
    int nt_x = 0, nt_y = 0;
    // fused x and z: one CTA per (y, component)
    void (*a)(PassArgs) = nullptr;
    void (*c)(PassArgs) = nullptr;
    void (*ab)(PassArgs) = nullptr;  // batched (grid.y extended by the instance count)
    void (*cb)(PassArgs) = nullptr;
    size_t smem_ac = 0;
    int nt_ac = 0;
    // bytes of pass C's x/z scratch (Xs and the exchange lines), which its
    // z phase can borrow for a TMA-loaded spectrum slab
    size_t ac_scratch = 0;
    bool slab_ok = false;  // pass C can take its z input as one slab
};
}  // namespace umag

struct umag_demag {
    umag::Passes fast;
    bool use_lines = false;  // line transforms; else the runtime-planned passes of demag.cu
    // P: the reference's padded sizes (mag/demagkernel.go:404-420), which
    // the real-space kernel and the spectrum are reported on.  F: the sizes
    // transformed here: P, or for line transforms the shortest supported
    // ones that hold the mesh
    int N[3], P[3], F[3];
    int pbc[3] = {0, 0, 0};  // PBC repetitions per axis (mag/demagkernel.go:339-355); padded size = N there
    double cell[3];
    int arad, zero_self;
    int kind = 0;           // real-space kernel: 0 Newell, 1 brute force, 2 caller-supplied
    double accuracy = 6.0;  // brute force: DemagAccuracy (engine/demag.go:25)
    int M, Hx, HxP, Lx, WB;
    bool is2d;
    umag::FftLine<float> fx, fy, fz;  // x: length F[0]/2 (packed real), y: F[1], z: F[2]
    std::vector<float2*> tw_dev;
    std::vector<float> ref_spec[6];   // caller-supplied kernels with F != P: the spectrum on P
    float2* twr = nullptr;            // exp(-2 pi i k / F[0]), k in [0, F[0]/2)
    float2* spec = nullptr;           // 3 * F[2] * Ny * Lx
    float* K[6] = {};                 // xx yy zz yz xz xy (yz, xz NULL in 2D)
    size_t Kn = 0;  // floats per kernel array (Kp * (F[1]/2+1) * (F[2]/2+1))
    int Kp = 0;     // row pitch: Px/2+1 rounded up to 4 floats (16-byte rows)
    CUtensorMap* slab_map = nullptr;  // device copy: pass C's (y, component) slabs of spec
};

namespace umag {

struct PassArgs {
    int Nx, Ny, Nz, Px, Py, Pz, M, Hx, HxP, Lx, WB;  // P: the transformed sizes (umag_demag::F)
    FftLine<float> fx, fy, fz;
    const float2* twr;
    float2* spec;
    const float* K[6];
    int Kp;  // row pitch (floats) of the kernel arrays: Hx padded to 4 in plans, Hx for caller-owned spectra
    // kernel arrays in 4-column blocks [kz][kx/4][ky][kx%4] (else rows
    // [kz][ky][kx] of pitch Kp).  The line passes hold the spectrum in
    // 4-column blocks [c][kz][kx/4][y][kx%4], the runtime-planned ones in rows
    int Kblocked;
    // batched launches: per-instance strides of the spectrum scratch (float2),
    // of the field output (floats) and of the controller structs holding
    // m_ind / m_ind_w / active (bytes); per-instance Ms (NULL: Ms_mul for all)
    long spec_stride, b_stride, ctl_stride;
    const float* ms_mul_b;
    const float* m[3];
    // engine use: magnetisation read through a device-side slot
    // (m_sel ? *m_ind_w : *m_ind) + c*ncell, and a device flag that turns a
    // skipped step into no-ops.  NULL for the plain device-op API.
    float* const* m_ind;
    float* const* m_ind_w;
    int m_sel;
    // the kernel before the first pass leaves the slots and the flag alone, so
    // they can be read while it runs (later passes always can)
    int early;
    int ncell;
    const int* active;
    const float* vol;
    const float* Ms;
    float Ms_mul;
    float* B[3];
    // tensor map (device memory) of the blocked spectrum viewed as
    // (8 floats, y, kx/4, kz, component): pass C loads the slab of one
    // (y, component) with one bulk tensor copy; NULL: plain loads
    const CUtensorMap* slab_map;
    // engine use: the controller's status word (instance ib at fault +
    // ib * ctl_stride bytes), set to 7 when a pass gives up waiting for a
    // bulk copy; NULL for the plain device-op API, which counts such
    // timeouts in *timeouts instead
    int* fault;
    unsigned* timeouts;  // device counter of bulk copies that timed out
};

int demag_new_newell(int Nx, int Ny, int Nz, const int pbc[3], double cx, double cy, double cz, int arad,
                     int zero_self, umag_demag** out);
int demag_new_from_kernel(int Nx, int Ny, int Nz, const double* const kern[6], umag_demag** out);
int demag_new_brute(int Nx, int Ny, int Nz, const int pbc[3], double cx, double cy, double cz, double accuracy,
                    umag_demag** out);
// brute-force real-space kernel (brute.cu) into six device arrays of the padded grid P
int build_brute(const umag_demag* d, const int P[3], double accuracy, double* Kr[6], cudaStream_t st);
int demag_exec(umag_demag* d, float* Bx, float* By, float* Bz, const float* mx, const float* my, const float* mz,
               const float* vol, const float* Ms, float Ms_mul, int pass = -1);
int demag_get_kernel(umag_demag* d, double* const host[6]);
int demag_get_spectrum(umag_demag* d, float* const host[6]);
void demag_free(umag_demag* d);
void fill_pass_args(const umag_demag* d, PassArgs& a);
// overlap: the kernel queued before it calls pdl_wait (common.cuh)
int demag_launch(const umag_demag* d, const PassArgs& a, cudaStream_t st, bool overlap = false);
// kernels that demag_launch queues
int demag_launches(const umag_demag* d);
int demag_launch_batch(const umag_demag* d, const PassArgs& a, int nb, cudaStream_t st, bool overlap = false);
// the line kernels for mesh N and their sizes F (with the fused x/z passes of F;
// exact: of the reference's padded sizes only); false: no such lengths
bool lines_select(const int N[3], const int pbc[3], int F[3], Passes& f, bool exact);
bool lines_x(int M, int npar, Passes& f);
bool lines_y(int L, int npar, Passes& f);
bool lines_z(int H, int npar, Passes& f);
bool fused_select(int M, int Pz, Passes& f);
// shared-memory opt-in of one pass kernel, once per device; thread-safe
int pass_attrs(void (*k)(PassArgs));
int passes_attrs(const Passes& f);
// meshes the batched ensembles and the no-alloc entry point take
bool listed_mesh(const int N[3], const int P[3]);
// no-alloc entry point: load its module on the current device (umag_init)
int noalloc_preload();
// bulk-copy waits of the demag passes that gave up since the counter was
// last cleared (demag_fast.cu); demag_exec reports them as an error
int demag_timeouts_ptr(unsigned** out);
int demag_slab_timeouts(unsigned* out, cudaStream_t st);
int demag_set_slab_timeouts(unsigned v);

}  // namespace umag
