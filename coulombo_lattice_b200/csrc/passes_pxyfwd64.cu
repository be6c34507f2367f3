// Launchers of the quadrant plane passes (plane_w.cuh, plane_xy.cuh) for planes of two lengths, forward, in FP64.
#include <algorithm>

#include "passes_impl.cuh"
#include "plane_xy.cuh"

namespace clp {

template <>
bool pfwd_xy<double>(cudaStream_t s, const cx<double>* rho, long long rho_stride, const int* row_ptr, const unsigned long long* row_mask,
                    cx<double>* buf, long long M, const cx<double>* twx, const cx<double>* twy, int nx, int ny, int nz,
                    int cnt) {
    return clk::pw::with_plane_w(nx, [&](auto tag) {
        using P = clk::pw::PlaneXY<double, decltype(tag)::r1, decltype(tag)::r2, true>;
        auto kern = clk::pw::k_pfwd_xy<double, decltype(tag)::r1, decltype(tag)::r2>;
        set_smem(kern, 227 * 1024);
        kern<<<dim3((unsigned)nz, plane_groups(nz, cnt, P::resident(ny))), P::THREADS, P::smem(ny), s>>>(
            rho, rho_stride, row_ptr, row_mask, buf, M, twx, twy, ny, cnt);
    });
}

}  // namespace clp
