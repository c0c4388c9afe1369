// demag_lines_yp.cu -- instantiations of the y line kernels (demag_lines.cuh).
#include "demag_lines.cuh"

namespace umag {

template <int L> static void fill_y(Passes& f) {
    using S = YShape<L, 1>;
    f.y = k_y<L, 1>;
    f.nt_y = S::NT;
    f.smem_y3 = S::smem(6);
    f.smem_y2 = S::smem(4);
}
bool lines_y_periodic(int L, Passes& f) {
    switch (L) {
#define Y(l) case l: fill_y<l>(f); return true;
        Y(4) Y(6) Y(8) Y(10) Y(12) Y(16) Y(20) Y(24) Y(30) Y(32) Y(40) Y(48) Y(50) Y(60) Y(64) Y(80) Y(96)
        Y(100) Y(120) Y(128) Y(160) Y(192) Y(200) Y(256) Y(320) Y(384) Y(512) Y(640) Y(768) Y(1024)
#undef Y
    default: return false;
    }
}

}  // namespace umag
