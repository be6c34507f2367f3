// Which (left, right) pairs of densities a Gram launch computes, as tiles.
//
// The steps of a request pair only some densities: with "eeee,hhhh,ehhe,eheh" the densities of two
// electrons or two holes meet each other but never those of an electron and a hole.  The connected
// components of the pairing are blocks of the Gram; only their tiles are computed.  Within a block
// whose left and right densities are the same, in the same order, the Gram of the whole convolution is
// symmetric (the Coulomb kernel is real and even: sum V_l rho_r = sum V_r rho_l, with the re x im and
// im x re sums exchanged), so tiles entirely above the diagonal are left out and a step reads the entry
// (larger, smaller).
#pragma once

#ifdef __CUDACC__
#define CLG_HD __host__ __device__
#else
#define CLG_HD
#endif

namespace clk {

constexpr int kGramBlocks = 8;

struct GramBlock {
    int l0, nl, r0, nr;  // left rows [l0, l0 + nl), right columns [r0, r0 + nr)
    int sym;             // same densities on both sides, in the same order
};

struct GramTile {
    int l0, nl, r0, nr;  // this tile's rows and columns
    int diag;            // symmetric block: index of row 0 minus index of column 0; pairs (l, r) with
                         // l + diag < r are not needed.  Otherwise large.
};

// The blocks of a launch, cut into tiles of at most wl[b] x wr[b] densities (equal widths but for the last).
struct GramTiles {
    int n, ldr;  // blocks; columns of the result
    GramBlock b[kGramBlocks];
    int wl[kGramBlocks], wr[kGramBlocks];
};

// Column tiles of row tile i in block b.
CLG_HD inline int gram_row_tiles(const GramTiles& g, int b, int i) {
    const GramBlock& k = g.b[b];
    int cols = k.nr;
    if (k.sym) {
        const int end = (i + 1) * g.wl[b];
        cols = end < k.nr ? end : k.nr;  // columns up to the tile's last row
    }
    return (cols + g.wr[b] - 1) / g.wr[b];
}

// Tile t of the launch in block, row, column order; returns the number of tiles when t < 0.
CLG_HD inline int gram_tile(const GramTiles& g, int t, GramTile* out) {
    int seen = 0;
    for (int b = 0; b < g.n; ++b) {
        const GramBlock& k = g.b[b];
        for (int i = 0; i * g.wl[b] < k.nl; ++i) {
            const int c = gram_row_tiles(g, b, i);
            if (t >= seen && t < seen + c) {
                const int j = t - seen, l = i * g.wl[b], r = j * g.wr[b];
                out->l0 = k.l0 + l;
                out->nl = g.wl[b] < k.nl - l ? g.wl[b] : k.nl - l;
                out->r0 = k.r0 + r;
                out->nr = g.wr[b] < k.nr - r ? g.wr[b] : k.nr - r;
                out->diag = k.sym ? l - r : 1 << 28;
                return seen;
            }
            seen += c;
        }
    }
    return seen;
}

// Tiles of at most max_l x max_r densities, their widths multiples of `step`.
inline GramTiles gram_tiles(const GramBlock* b, int n, int nr, int max_l, int max_r, int step) {
    const auto width = [step](int count, int most) {
        const int tiles = (count + most - 1) / most;
        const int w = (count + tiles - 1) / tiles;
        return (w + step - 1) / step * step;
    };
    GramTiles g{};
    g.n = n;
    g.ldr = nr;
    for (int i = 0; i < n; ++i) {
        g.b[i] = b[i];
        g.wl[i] = width(b[i].nl, max_l);
        g.wr[i] = width(b[i].nr, max_r);
    }
    return g;
}
inline int gram_tile_count(const GramTiles& g) { return gram_tile(g, -1, nullptr); }

}  // namespace clk
