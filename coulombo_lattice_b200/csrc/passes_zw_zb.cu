// Class-mixing z pass of the zinc-blende class set (zmix_wht.cuh) in FP32.
#include "passes_zw_impl.cuh"

namespace clp {

template <>
bool zw_zb<float>(cudaStream_t s, cx<float>* buf, long long stride, const cx<float>* tw, const clk::Quad<float>* tab,
             const cx<float>* col, const cx<float>* zph, long long nxy, int nz, int cnt) {
    return zw_launch<clk::kZwZb, float>(s, buf, stride, tw, tab, col, zph, nxy, nz, cnt);
}
bool zw_zb_supported(int nz) {
    return clk::with_zw_split<clk::kZwZb>(nz, [](auto) {});
}

}  // namespace clp
