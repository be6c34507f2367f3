// Launchers of the quadrant plane passes (plane_w.cuh, plane_xy.cuh) for square planes in FP64.
#include <algorithm>

#include "passes_impl.cuh"
#include "plane_w.cuh"

namespace clp {

template <>
bool pfwd<double>(cudaStream_t s, const cx<double>* rho, long long rho_stride, const int* row_ptr, const unsigned long long* row_mask,
                 cx<double>* buf, long long M, const cx<double>* tw, int n, int nz, int cnt) {
    return clk::pw::with_plane_w(n, [&](auto tag) {
        using L = clk::pw::PlaneW<double, decltype(tag)::r1, decltype(tag)::r2, true>;
        if constexpr (L::smem <= 227 * 1024) {
            auto kern = clk::pw::k_pfwd<double, decltype(tag)::r1, decltype(tag)::r2>;
            set_smem(kern, L::smem);
            kern<<<dim3((unsigned)nz, plane_groups(nz, cnt, L::MIN)), L::THREADS, L::smem, s>>>(
                rho, rho_stride, row_ptr, row_mask, buf, M, tw, cnt);
        }
    });
}

template <>
bool pinv<double>(cudaStream_t s, const cx<double>* buf, long long M, const cx<double>* tw, const int* row_ptr,
                 const unsigned long long* row_mask, cx<double>* out, long long o_stride, int n, int nz, int cnt) {
    return clk::pw::with_plane_w(n, [&](auto tag) {
        using L = clk::pw::PlaneW<double, decltype(tag)::r1, decltype(tag)::r2, false>;
        if constexpr (L::smem <= 227 * 1024) {
            auto kern = clk::pw::k_pinv<double, decltype(tag)::r1, decltype(tag)::r2>;
            set_smem(kern, L::smem);
            kern<<<dim3((unsigned)nz, plane_groups(nz, cnt, L::MIN)), L::THREADS, L::smem, s>>>(
                buf, M, tw, row_ptr, row_mask, out, o_stride, cnt);
        }
    });
}

}  // namespace clp
