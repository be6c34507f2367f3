// Launchers of the quadrant plane passes (plane_w.cuh).
#include <algorithm>

#include "passes_impl.cuh"
#include "plane_w.cuh"

namespace clp {

bool quadrant_supported(int nx, int ny) {
    return clk::pw::with_plane_w(nx, [](auto) {}) && clk::pw::with_plane_w(ny, [](auto) {});
}

bool pfwd(cudaStream_t s, const cx<float>* rho, long long rho_stride, const int* row_ptr, const int* cell,
          cx<float>* buf, long long M, const cx<float>* tw, int n, int nz, int cnt) {
    return clk::pw::with_plane_w(n, [&](auto tag) {
        using L = clk::pw::PlaneW<decltype(tag)::r1, decltype(tag)::r2, true>;
        auto kern = clk::pw::k_pfwd<decltype(tag)::r1, decltype(tag)::r2>;
        set_smem(kern, L::smem);
        kern<<<dim3((unsigned)nz, plane_groups(nz, cnt, L::MIN)), L::THREADS, L::smem, s>>>(rho, rho_stride, row_ptr,
                                                                                            cell, buf, M, tw, cnt);
    });
}

bool pinv(cudaStream_t s, const cx<float>* buf, long long M, const cx<float>* tw, const int* row_ptr, const int* cell,
          cx<float>* out, long long o_stride, int n, int nz, int cnt) {
    return clk::pw::with_plane_w(n, [&](auto tag) {
        using L = clk::pw::PlaneW<decltype(tag)::r1, decltype(tag)::r2, false>;
        auto kern = clk::pw::k_pinv<decltype(tag)::r1, decltype(tag)::r2>;
        set_smem(kern, L::smem);
        kern<<<dim3((unsigned)nz, plane_groups(nz, cnt, L::MIN)), L::THREADS, L::smem, s>>>(buf, M, tw, row_ptr, cell,
                                                                                            out, o_stride, cnt);
    });
}

}  // namespace clp
