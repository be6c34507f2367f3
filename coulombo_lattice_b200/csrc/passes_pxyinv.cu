// Launchers of the quadrant plane passes (plane_w.cuh, plane_xy.cuh) for planes of two lengths, inverse, in FP32.
#include <algorithm>

#include "passes_impl.cuh"
#include "plane_xy.cuh"

namespace clp {

template <>
bool pinv_xy<float>(cudaStream_t s, const cx<float>* buf, long long M, const cx<float>* twx, const cx<float>* twy,
                    const int* row_ptr, const unsigned long long* row_mask, cx<float>* out, long long o_stride, int nx, int ny, int nz,
                    int cnt) {
    return clk::pw::with_plane_w(nx, [&](auto tag) {
        using P = clk::pw::PlaneXY<float, decltype(tag)::r1, decltype(tag)::r2, false>;
        auto kern = clk::pw::k_pinv_xy<float, decltype(tag)::r1, decltype(tag)::r2>;
        set_smem(kern, 227 * 1024);
        kern<<<dim3((unsigned)nz, plane_groups(nz, cnt, P::resident(ny))), P::THREADS, P::smem(ny), s>>>(
            buf, M, twx, twy, row_ptr, row_mask, out, o_stride, ny, cnt);
    });
}

}  // namespace clp
