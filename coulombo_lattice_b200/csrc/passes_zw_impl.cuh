// Launcher body of the class-mixing z pass (zmix_wht.cuh); included by passes_zw_zb.cu and
// passes_zw_pair.cu (one class set per translation unit, compiled in parallel).
#pragma once

#include <algorithm>

#include "passes_impl.cuh"
#include "zmix_wht.cuh"

namespace clp {

namespace {

// Density groups (gridDim.y) of a launch over `blocks` column blocks: the count whose modelled span is
// shortest -- waves of blocks over the resident slots, times the densities a warp group runs plus its
// setup (the table of its columns and the first staging, about one density).  128-point lines, 36
// densities: 1.85 ms with one group, 1.96 with two; 64-point, 400 densities: 2.37 with one (3.5 waves),
// 2.10 with two.
unsigned zw_density_groups(long long blocks, int cnt, int groups, int blocks_per_sm) {
    const long long slots = 148LL * blocks_per_sm;
    unsigned best = 1;
    double best_t = 1e300;
    for (int y = 1; y <= cnt; ++y) {
        const int per = (cnt + y - 1) / y;
        if ((long long)(y - 1) * per >= cnt) continue;  // a group would be empty
        const long long waves = (blocks * y + slots - 1) / slots;
        const double t = (double)waves * ((per + groups - 1) / groups + 1);
        if (t < best_t) {
            best_t = t;
            best = (unsigned)y;
        }
    }
    return best;
}

template <int SET, typename T>
bool zw_launch(cudaStream_t s, cx<T>* buf, long long stride, const cx<T>* tw, const clk::Quad<T>* tab,
               const cx<T>* col, const cx<T>* zph, long long nxy, int nz, int cnt) {
    return clk::with_zw_split<SET>(nz, [&](auto tag) {
        using Tag = decltype(tag);
        using Lay = clk::ZwLayout<T, SET, Tag::r1, Tag::r2>;
        const long long blocks = (nxy + Lay::L - 1) / Lay::L;
        constexpr int per_sm = Lay::resident(Lay::G) / (Lay::NT * Lay::G);
        const unsigned y = zw_density_groups(blocks, cnt, Lay::G, per_sm);
        const int groups = std::min<int>(Lay::G, (cnt + (int)y - 1) / (int)y);
        auto kern = clk::k_zw<T, SET, Tag::r1, Tag::r2>;
        set_smem(kern, Lay::smem(Lay::G));
        kern<<<dim3((unsigned)blocks, y), Lay::NT * groups, Lay::smem(groups), s>>>(buf, stride, tw, tab, col, zph,
                                                                                   nxy, cnt);
    });
}

}  // namespace

}  // namespace clp
