// demag_lines_x.cu -- instantiations of the x line kernels (demag_lines.cuh).
#include "demag_lines.cuh"

namespace umag {

template <int L, int NPAR> static void fill_x(Passes& f) {
    f.xf = k_x_fwd<L, NPAR>;
    f.xi = k_x_inv<L, NPAR>;
    f.nt_x = XShape<L, NPAR>::NT;
    f.smem_x = XShape<L, NPAR>::smem;
}
bool lines_x(int L, int npar, Passes& f) {
    switch (L) {
#define X(l)                                  \
    case l:                                   \
        if (npar == 2) fill_x<l, 2>(f);       \
        else fill_x<l, 1>(f);                 \
        return true;
        X(4) X(6) X(8) X(10) X(12) X(16) X(20) X(24) X(30) X(32) X(40) X(48) X(50) X(60) X(64) X(80) X(96)
        X(100) X(120) X(128) X(160) X(192) X(200) X(256) X(320) X(384) X(512)
#undef X
    default: return false;
    }
}

}  // namespace umag
