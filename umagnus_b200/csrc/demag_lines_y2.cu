// demag_lines_y2.cu -- instantiations of the y line kernels (demag_lines.cuh).
#include "demag_lines.cuh"

namespace umag {

template <int L> static void fill_y(Passes& f) {
    using S = YShape<L, 2>;
    f.y = k_y<L, 2>;
    f.nt_y = S::NT;
    f.smem_y3 = S::smem(6);
    f.smem_y2 = S::smem(4);
}
bool lines_y_open2(int L, Passes& f) {
    switch (L) {
#define Y(l) case l: fill_y<l>(f); return true;
        Y(8) Y(16) Y(30) Y(48) Y(64) Y(100) Y(160) Y(256) Y(512) Y(1024)
#undef Y
    default: return false;
    }
}

}  // namespace umag
