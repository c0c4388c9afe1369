// demag_lines_z.cu -- instantiations of the z line kernels (demag_lines.cuh).
#include "demag_lines.cuh"

namespace umag {

template <int H, int NPAR> static void fill_z(Passes& f) {
    f.zf = k_z_fwd<H, NPAR>;
    f.zi = k_z_inv<H, NPAR>;
}
bool lines_z(int H, int npar, Passes& f) {
    switch (H) {
#define Z(h)                                  \
    case h:                                   \
        if (npar == 2) fill_z<h, 2>(f);       \
        else fill_z<h, 1>(f);                 \
        return true;
        Z(2) Z(3) Z(4) Z(5) Z(6) Z(8) Z(10) Z(12) Z(16) Z(20) Z(24) Z(32)
#undef Z
    default: return false;
    }
}

// open y lines are spread over three files to compile in parallel
bool lines_y_open0(int L, Passes& f);
bool lines_y_open1(int L, Passes& f);
bool lines_y_open2(int L, Passes& f);
bool lines_y_periodic(int L, Passes& f);
bool lines_y(int L, int npar, Passes& f) {
    if (npar == 1) return lines_y_periodic(L, f);
    return lines_y_open0(L, f) || lines_y_open1(L, f) || lines_y_open2(L, f);
}

}  // namespace umag
