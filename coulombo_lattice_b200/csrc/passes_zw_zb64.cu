// Class-mixing z pass of the zinc-blende class set (zmix_wht.cuh) in FP64.
#include "passes_zw_impl.cuh"

namespace clp {

template <>
bool zw_zb<double>(cudaStream_t s, cx<double>* buf, long long stride, const cx<double>* tw, const clk::Quad<double>* tab,
             const cx<double>* col, const cx<double>* zph, long long nxy, int nz, int cnt) {
    return zw_launch<clk::kZwZb, double>(s, buf, stride, tw, tab, col, zph, nxy, nz, cnt);
}

}  // namespace clp
