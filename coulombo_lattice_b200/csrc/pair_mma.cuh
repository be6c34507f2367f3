// Pair densities at the atoms on the FP64 tensor cores, for requests over at most 40 states.
//
// For one atom the products rho_ij = sum_o conj(c_i[o]) c_j[o] (Product.cpp:16-30) of S states are the
// lower triangle of a Hermitian S x S matrix: with R, X the real and imaginary parts of the atom's S x
// n_orb coefficients,
//     Re = R R^T + X X^T,   Im = R X^T - X R^T.
// States go in blocks of 8; one or four warps take an atom and form its 8 x 8 tiles (bi, bj), bj <= bi,
// with mma.sync m8n8k4 .f64 over 4 orbitals a step.  The fragment of the left operand (row = lane / 4, k =
// lane % 4) is that of the right one (column = lane / 4), so a step needs one 16-byte shared load per
// block and lane and 4 MMAs a tile.  FOLD: 3 on the diagonal, where X R^T is the transpose of R X^T
// (exchanged once an atom by shuffles: a gain from about 4 steps, 16 orbitals, on).  Products are exact FP64 FMAs summed in FP64, rounded once to RT.
// Up to 4 states leave most of a tile empty, so it takes 2, 4 or 8 atoms of 4, 2 or 1 rows each: the products
// of one atom are a block on the tile's diagonal, the rest is not used.
//
// A thread block works through batches of `at` consecutive atoms: the batch's coefficients, at n_orb
// contiguous values a state, go to shared memory with 16-byte cp.async, two batches deep (states 64
// bytes off a 128-byte row: the lanes of a fragment hit distinct banks), the products come back through
// shared memory as [product][atom], two of them in turn, and leave in runs of `at` atoms: one barrier a
// batch.  SLICED: where one atom a warp group does not fit (72 orbitals at 12 states, 108 at 8), a batch comes in
// slices of orbitals and a warp keeps its atom's sums over them.
//
// Bound: HBM at 8 states, the FP64 tensor pipe and the shared-memory traffic above.  Measured on a B200
// against the kernels it replaced (register products from shared memory at up to 12 states, 4 x 4-state
// tiles above), 20 orbitals: 8 states, 2,097,152 atoms, 1.29 -> 1.01 ms (5.9 TB/s); 12 states, 110,592
// atoms, 0.189 -> 0.130 ms; 40 states, 262,144 atoms, 3.53 -> 2.04 ms.  Fragments loaded straight from HBM,
// five steps ahead: 1.50, 0.196 and 2.13 ms.
// With one atom a tile, 2 states, 20 orbitals, 110,592 atoms took 0.051 ms and 4 states 0.053 (the register kernel
// 0.022 and 0.047); several share one: 0.023 and 0.037.  Orbitals in slices, 32,768 atoms: 12 states, 80 orbitals
// 0.147 ms (register kernel 0.231, tiles 1.05); 8 and 112, 0.102 (0.135 and 0.87); 40 and 40, 0.54 (tiles 1.11).
#pragma once

#include <cstdint>

#include "fft.cuh"
#include "kernels.cuh"

namespace clk {
namespace pm {

constexpr int MAX_BLOCKS = 5;  // 40 states

// Warps a block, warps that share an atom's tiles, and blocks an SM (registers): up to 24 states a warp
// holds all its atom's tiles (6, 48 registers of sums); 10 and 15 tiles go over four warps.
__host__ __device__ constexpr int warps(int nb) { return nb <= 3 ? 8 : 16; }
__host__ __device__ constexpr int warps_per_atom(int nb) { return nb <= 3 ? 1 : 4; }
__host__ __device__ constexpr int min_blocks(int nb) { return nb == 1 ? 4 : nb == 2 ? 3 : nb == 3 ? 2 : 1; }

struct PairMmaArgs {
    const cx<double>* coeff;    // [state][atom][orbital]
    int n_orb;
    long long n;                // atoms
    const int* prod;            // [8 NB][8 NB]: density row of product (i, j), i >= j; -1 not requested
    int np;                     // density rows
    int at, at_log2;            // atoms a batch: a power of two, at least warps / warps_per_atom tiles
    int rows_log2;              // rows of a tile an atom takes: 8 but for at most 4 states
    int slice_log2;             // SLICED: orbitals a slice
    int state_pitch;            // elements between the states of a staged batch
    int n_used;
    int state[8 * MAX_BLOCKS];  // coefficient row of each used state, ascending
};

// Elements between the states of a staged batch of n_orb values an atom: 64 bytes off a multiple of 128.
inline int state_pitch(int at, int n_orb) {
    const int e = at * n_orb;
    return e + (12 - e % 8) % 8;
}
template <typename RT>
size_t pair_mma_smem(int nb, int n_used, int pitch, int np, int at) {
    const int tiles = nb * (nb + 1) / 2;
    return sizeof(cx<double>) * (size_t)2 * n_used * pitch + 2 * sizeof(cx<RT>) * (size_t)np * (at + 1) +
           sizeof(short) * 64 * tiles;
}

__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

__host__ __device__ constexpr int tile_row(int t) {
    int bi = 0;
    while ((bi + 1) * (bi + 2) / 2 <= t) ++bi;
    return bi;
}
__host__ __device__ constexpr int tile_col(int t) { return t - tile_row(t) * (tile_row(t) + 1) / 2; }

// The sums of a warp's tiles [H TH, ...) of one atom (or of the atoms that share a tile).
template <int NB, int WPA>
struct Sums {
    static constexpr int T = NB * (NB + 1) / 2, TH = (T + WPA - 1) / WPA;
    double re[TH][2], im[TH][2];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int t = 0; t < TH; ++t) re[t][0] = re[t][1] = im[t][0] = im[t][1] = 0.0;
    }
};
template <int NB, int WPA, int H>
struct Part {
    static constexpr int T = Sums<NB, WPA>::T, TH = Sums<NB, WPA>::TH, T0 = H * TH, N = (T0 + TH < T ? T0 + TH : T) - T0;
};

// Adds n_orb orbitals: c is the lane's first of state row 0 of block 0 (staged).
template <int NB, int WPA, int H, bool FOLD>
__device__ __forceinline__ void add_orbitals(Sums<NB, WPA>& s, const cx<double>* c, int block_pitch, int n_orb, int tig,
                                             unsigned have) {
    constexpr int T0 = Part<NB, WPA, H>::T0, N = Part<NB, WPA, H>::N;
#pragma unroll 2
    for (int o = 0; o < n_orb; o += 4) {
        cx<double> v[NB];
#pragma unroll
        for (int b = 0; b < NB; ++b)
            v[b] = (o + tig < n_orb && ((have >> b) & 1u)) ? c[(size_t)b * block_pitch + o] : mk(0.0, 0.0);
#pragma unroll
        for (int t = 0; t < N; ++t) {
            const int bi = tile_row(T0 + t), bj = tile_col(T0 + t);
            mma_f64(s.re[t], v[bi].re, v[bj].re);
            mma_f64(s.im[t], v[bi].re, v[bj].im);
        }
#pragma unroll
        for (int t = 0; t < N; ++t) {
            const int bi = tile_row(T0 + t), bj = tile_col(T0 + t);
            mma_f64(s.re[t], v[bi].im, v[bj].im);
            if (!FOLD || bi != bj) mma_f64(s.im[t], -v[bi].im, v[bj].re);
        }
    }
}

// Rounds the products and puts them at out[product * out_pitch] (out: the lane's atom).
template <int NB, int WPA, int H, bool FOLD, typename RT>
__device__ __forceinline__ void put_products(Sums<NB, WPA>& s, int tig, const short* row, int lane, cx<RT>* out,
                                             int out_pitch) {
    constexpr int T0 = Part<NB, WPA, H>::T0, N = Part<NB, WPA, H>::N;
#pragma unroll
    for (int t = 0; t < N; ++t) {
        if (FOLD && tile_row(T0 + t) == tile_col(T0 + t)) {
            // X R^T of a diagonal tile is the transpose of its R X^T: element (j, i) is held by lane 4 j +
            // i / 2 as its (i mod 2)-th
            double turned[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int from = 4 * (2 * tig + h) + (lane >> 3);
                const double e0 = __shfl_sync(0xffffffffu, s.im[t][0], from), e1 = __shfl_sync(0xffffffffu, s.im[t][1], from);
                turned[h] = (lane >> 2) & 1 ? e1 : e0;
            }
            s.im[t][0] -= turned[0];
            s.im[t][1] -= turned[1];
        }
        const short2 r = *reinterpret_cast<const short2*>(row + ((T0 + t) * 32 + lane) * 2);
        if (r.x >= 0) out[r.x * out_pitch] = narrow<RT>(mk(s.re[t][0], s.im[t][0]));
        if (r.y >= 0) out[r.y * out_pitch] = narrow<RT>(mk(s.re[t][1], s.im[t][1]));
    }
}

// f(H as an integral constant) for the warp's part of an atom's tiles.
template <int H>
struct PartTag {
    static constexpr int value = H;
};
template <int WPA, typename F>
__device__ __forceinline__ void warp_part(int warp, F&& f) {
    if constexpr (WPA == 1) {
        f(PartTag<0>{});
    } else {
        switch (warp % WPA) {
            case 0: f(PartTag<0>{}); break;
            case 1: f(PartTag<1>{}); break;
            case 2: f(PartTag<2>{}); break;
            default: f(PartTag<3>{}); break;
        }
    }
}

// PACKED: at most 4 states, several atoms a tile.
template <int NB, bool PACKED, bool FOLD, bool SLICED, typename RT>
__global__ void __launch_bounds__(32 * warps(NB), min_blocks(NB))
    k_pair_mma(const PairMmaArgs g, cx<RT>* __restrict__ rho) {
    constexpr int T = NB * (NB + 1) / 2, WARPS = warps(NB), THREADS = 32 * WARPS, WPA = warps_per_atom(NB), S = 8 * NB;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cx<double>* in = reinterpret_cast<cx<double>*>(smem_raw);  // [2][state][state_pitch]
    const int in_stage = g.n_used * g.state_pitch;
    cx<RT>* out = reinterpret_cast<cx<RT>*>(in + (size_t)2 * in_stage);  // [2][product][at + 1]
    const int pitch = g.at + 1;
    short* row = reinterpret_cast<short*>(out + (size_t)2 * g.np * pitch);  // [tile][lane][2]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int grp = lane >> 2, tig = lane & 3;
    const int rl = PACKED ? g.rows_log2 : 3, per_tile = 8 >> rl;  // atoms a tile
    const long long batches = (g.n + g.at - 1) / g.at;
    const int slice = SLICED ? 1 << g.slice_log2 : g.n_orb;
    const int slices = SLICED ? (g.n_orb + slice - 1) >> g.slice_log2 : 1;
    // the copies of a state go to WARPS / n_used warps where that is more than one
    const int sharers = g.n_used < WARPS ? WARPS / g.n_used : 1;
    const auto copy_in = [&](long long b, int sl, int stage) {
        if (b < batches) {
            const long long a0 = b * g.at;
            const int atoms = (int)min((long long)g.at, g.n - a0);
            for (int w = warp; w < g.n_used * sharers; w += WARPS) {
                const int s = sharers == 1 ? w : w % g.n_used, first = sharers == 1 ? lane : lane + 32 * (w / g.n_used);
                const cx<double>* src = g.coeff + ((long long)g.state[s] * g.n + a0) * g.n_orb;
                cx<double>* dst = in + (size_t)stage * in_stage + (size_t)s * g.state_pitch;
                if (SLICED) {
                    for (int e = first; e < atoms << g.slice_log2; e += 32 * sharers) {
                        const int a = e >> g.slice_log2, o = (sl << g.slice_log2) + (e & (slice - 1));
                        if (o < g.n_orb) pd_cp_async16(dst + e, src + (long long)a * g.n_orb + o);
                    }
                } else {
                    for (int e = first; e < atoms * g.n_orb; e += 32 * sharers) pd_cp_async16(dst + e, src + e);
                }
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    long long b = blockIdx.x;
    copy_in(b, 0, 0);
    for (int e = threadIdx.x; e < T * 64; e += THREADS) {
        const int t = e / 64, l = e / 2 % 32, h = e % 2;
        int bi = 0;
        while ((bi + 1) * (bi + 2) / 2 <= t) ++bi;
        const int bj = t - bi * (bi + 1) / 2;
        const int i = 8 * bi + l / 4, j = 8 * bj + 2 * (l % 4) + h;
        if (!PACKED) {
            row[e] = (short)(i >= j ? g.prod[i * S + j] : -1);
        } else {
            const int m = (1 << rl) - 1;
            row[e] = (short)(i >> rl == j >> rl && i >= j ? g.prod[(i & m) * S + (j & m)] : -1);
        }
    }
    unsigned have = 0;  // blocks in which this lane's state exists
    const int mine = PACKED ? grp & ((1 << rl) - 1) : grp, own = PACKED ? grp >> rl : 0;  // its row, its atom
#pragma unroll
    for (int k = 0; k < NB; ++k)
        if (8 * k + mine < g.n_used) have |= 1u << k;
    const int bp = 8 * g.state_pitch;
    int stage = 0, turn = 0;
    for (; b < batches; b += gridDim.x) {
        cx<RT>* o = out + (size_t)(turn & 1) * g.np * pitch;
        Sums<NB, WPA> sums;
        if (SLICED) sums.clear();
#pragma unroll 1
        for (int sl = 0; sl < slices; ++sl) {
            // the slice has landed, everyone's copies are visible, and everyone is done with the one before: its
            // stage takes the next copy, and the out buffer of two batches ago has been stored
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            __syncthreads();
            if (sl == 0 && turn > 0) {  // the previous batch's products
                const long long a0 = (b - gridDim.x) * g.at;
                const cx<RT>* done = out + (size_t)((turn - 1) & 1) * g.np * pitch;
                for (int e = threadIdx.x; e < g.np * g.at; e += THREADS) {
                    const int p = e >> g.at_log2, k = e & (g.at - 1);
                    rho[(long long)p * g.n + a0 + k] = done[p * pitch + k];  // a whole batch: not the last one
                }
            }
            const bool more = sl + 1 < slices;
            copy_in(more ? b : b + gridDim.x, more ? sl + 1 : 0, stage ^ 1);
            const cx<double>* st = in + (size_t)stage * in_stage + (size_t)mine * g.state_pitch;
            if constexpr (SLICED) {
                const int a = warp / WPA * per_tile + own;  // at is what the warps take at a time
                const int count = min(slice, g.n_orb - (sl << g.slice_log2));
                warp_part<WPA>(warp, [&](auto part) {
                    constexpr int H = decltype(part)::value;
                    add_orbitals<NB, WPA, H, FOLD>(sums, st + (a << g.slice_log2) + tig, bp, count, tig, have);
                    if (!more) put_products<NB, WPA, H, FOLD, RT>(sums, tig, row, lane, o + a, pitch);
                });
            } else {
#pragma unroll 1
                for (int a0 = warp / WPA * per_tile; a0 < g.at; a0 += WARPS / WPA * per_tile) {
                    const int a = a0 + own;
                    warp_part<WPA>(warp, [&](auto part) {
                        constexpr int H = decltype(part)::value;
                        sums.clear();
                        add_orbitals<NB, WPA, H, FOLD>(sums, st + a * g.n_orb + tig, bp, g.n_orb, tig, have);
                        put_products<NB, WPA, H, FOLD, RT>(sums, tig, row, lane, o + a, pitch);
                    });
                }
            }
            stage ^= 1;
        }
        ++turn;
    }
    if (turn == 0) return;
    __syncthreads();
    const long long a0 = (b - gridDim.x) * g.at;
    const int last = (int)min((long long)g.at, g.n - a0);
    const cx<RT>* o = out + (size_t)((turn - 1) & 1) * g.np * pitch;
    for (int e = threadIdx.x; e < g.np * g.at; e += THREADS) {
        const int p = e >> g.at_log2, k = e & (g.at - 1);
        if (k < last) rho[(long long)p * g.n + a0 + k] = o[p * pitch + k];
    }
}

}  // namespace pm
}  // namespace clk
