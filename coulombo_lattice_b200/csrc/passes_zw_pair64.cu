// Class-mixing z pass of two-class sets (zmix_wht.cuh) in FP64.
#include "passes_zw_impl.cuh"

namespace clp {

template <>
bool zw_pair<double>(cudaStream_t s, cx<double>* buf, long long stride, const cx<double>* tw, const clk::Quad<double>* tab,
             long long nxy, int nz, int cnt) {
    return zw_launch<clk::kZwPair, double>(s, buf, stride, tw, tab, nullptr, nullptr, nxy, nz, cnt);
}

}  // namespace clp
