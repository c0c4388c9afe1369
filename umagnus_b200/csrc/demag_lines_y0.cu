// demag_lines_y0.cu -- instantiations of the y line kernels (demag_lines.cuh).
#include "demag_lines.cuh"

namespace umag {

template <int L> static void fill_y(Passes& f) {
    using S = YShape<L, 2>;
    f.y = k_y<L, 2>;
    f.nt_y = S::NT;
    f.smem_y3 = S::smem(6);
    f.smem_y2 = S::smem(4);
}
bool lines_y_open0(int L, Passes& f) {
    switch (L) {
#define Y(l) case l: fill_y<l>(f); return true;
        Y(4) Y(10) Y(20) Y(32) Y(50) Y(80) Y(120) Y(192) Y(320) Y(640)
#undef Y
    default: return false;
    }
}

}  // namespace umag
