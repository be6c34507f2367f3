// Launchers of the quadrant plane passes (plane_w.cuh, plane_xy.cuh) for planes of two lengths, inverse, in FP64.
#include <algorithm>

#include "passes_impl.cuh"
#include "plane_xy.cuh"

namespace clp {

template <>
bool pinv_xy<double>(cudaStream_t s, const cx<double>* buf, long long M, const cx<double>* twx, const cx<double>* twy,
                    const int* row_ptr, const unsigned long long* row_mask, cx<double>* out, long long o_stride, int nx, int ny, int nz,
                    int cnt) {
    return clk::pw::with_plane_w(nx, [&](auto tag) {
        using P = clk::pw::PlaneXY<double, decltype(tag)::r1, decltype(tag)::r2, false>;
        auto kern = clk::pw::k_pinv_xy<double, decltype(tag)::r1, decltype(tag)::r2>;
        set_smem(kern, 227 * 1024);
        kern<<<dim3((unsigned)nz, plane_groups(nz, cnt, P::resident(ny))), P::THREADS, P::smem(ny), s>>>(
            buf, M, twx, twy, row_ptr, row_mask, out, o_stride, ny, cnt);
    });
}

}  // namespace clp
