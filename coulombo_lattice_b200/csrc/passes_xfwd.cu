// Forward x-pass launchers (passes.hpp) in FP32.
#include "passes_impl.cuh"

namespace clp {
template bool xfwd<float>(cudaStream_t, Variant, const cx<float>*, long long, const int*, const int*, cx<float>*,
                          long long, const cx<float>*, const clk::RoundPhase&, int, int, int, int, int);
}  // namespace clp
