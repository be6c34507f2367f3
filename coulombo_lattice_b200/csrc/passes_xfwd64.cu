// Forward x-pass launchers (passes.hpp) in FP64.
#include "passes_impl.cuh"

namespace clp {
template bool xfwd<double>(cudaStream_t, Variant, const cx<double>*, long long, const int*, const int*, cx<double>*,
                           long long, const cx<double>*, const clk::RoundPhase&, int, int, int, int, int);
}  // namespace clp
