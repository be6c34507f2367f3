// Class-mixing z pass of two-class sets (zmix_wht.cuh) in FP32.
#include "passes_zw_impl.cuh"

namespace clp {

template <>
bool zw_pair<float>(cudaStream_t s, cx<float>* buf, long long stride, const cx<float>* tw, const clk::Quad<float>* tab,
             long long nxy, int nz, int cnt) {
    return zw_launch<clk::kZwPair, float>(s, buf, stride, tw, tab, nullptr, nullptr, nxy, nz, cnt);
}
bool zw_pair_supported(int nz) {
    return clk::with_zw_split<clk::kZwPair>(nz, [](auto) {});
}

}  // namespace clp
