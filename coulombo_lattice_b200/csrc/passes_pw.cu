// Launchers of the quadrant plane passes (plane_w.cuh, plane_xy.cuh) for square planes in FP32.
#include <algorithm>

#include "passes_impl.cuh"
#include "plane_xy.cuh"

namespace clp {

bool quadrant_supported(bool fp32, int nx, int ny) {
    bool fits = false;
    const bool x = clk::pw::with_plane_w(nx, [&](auto tag) {
        constexpr int H = decltype(tag)::r1, R2 = decltype(tag)::r2;
        const size_t most = 227 * 1024;
        if (fp32)
            fits = clk::pw::PlaneXY<float, H, R2, true>::smem(ny) <= most &&
                   clk::pw::PlaneXY<float, H, R2, false>::smem(ny) <= most;
        else
            fits = clk::pw::PlaneXY<double, H, R2, true>::smem(ny) <= most &&
                   clk::pw::PlaneXY<double, H, R2, false>::smem(ny) <= most;
    });
    return x && fits && clk::pw::with_plane_w(ny, [](auto) {});
}

template <>
bool pfwd<float>(cudaStream_t s, const cx<float>* rho, long long rho_stride, const int* row_ptr, const unsigned long long* row_mask,
                 cx<float>* buf, long long M, const cx<float>* tw, int n, int nz, int cnt) {
    return clk::pw::with_plane_w(n, [&](auto tag) {
        using L = clk::pw::PlaneW<float, decltype(tag)::r1, decltype(tag)::r2, true>;
        if constexpr (L::smem <= 227 * 1024) {
            auto kern = clk::pw::k_pfwd<float, decltype(tag)::r1, decltype(tag)::r2>;
            set_smem(kern, L::smem);
            kern<<<dim3((unsigned)nz, plane_groups(nz, cnt, L::MIN)), L::THREADS, L::smem, s>>>(
                rho, rho_stride, row_ptr, row_mask, buf, M, tw, cnt);
        }
    });
}

template <>
bool pinv<float>(cudaStream_t s, const cx<float>* buf, long long M, const cx<float>* tw, const int* row_ptr,
                 const unsigned long long* row_mask, cx<float>* out, long long o_stride, int n, int nz, int cnt) {
    return clk::pw::with_plane_w(n, [&](auto tag) {
        using L = clk::pw::PlaneW<float, decltype(tag)::r1, decltype(tag)::r2, false>;
        if constexpr (L::smem <= 227 * 1024) {
            auto kern = clk::pw::k_pinv<float, decltype(tag)::r1, decltype(tag)::r2>;
            set_smem(kern, L::smem);
            kern<<<dim3((unsigned)nz, plane_groups(nz, cnt, L::MIN)), L::THREADS, L::smem, s>>>(
                buf, M, tw, row_ptr, row_mask, out, o_stride, cnt);
        }
    });
}

}  // namespace clp
