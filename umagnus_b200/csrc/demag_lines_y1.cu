// demag_lines_y1.cu -- instantiations of the y line kernels (demag_lines.cuh).
#include "demag_lines.cuh"

namespace umag {

template <int L> static void fill_y(Passes& f) {
    using S = YShape<L, 2>;
    f.y = k_y<L, 2>;
    f.nt_y = S::NT;
    f.smem_y3 = S::smem(6);
    f.smem_y2 = S::smem(4);
}
bool lines_y_open1(int L, Passes& f) {
    switch (L) {
#define Y(l) case l: fill_y<l>(f); return true;
        Y(6) Y(12) Y(24) Y(40) Y(60) Y(96) Y(128) Y(200) Y(384) Y(768)
#undef Y
    default: return false;
    }
}

}  // namespace umag
