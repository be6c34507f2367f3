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
//
// A thread block works through batches of `at` consecutive atoms: the batch's coefficients, at n_orb
// contiguous values a state, go to shared memory with 16-byte cp.async `stages` batches deep (states 64
// bytes off a 128-byte row: the lanes of a fragment hit distinct banks), the products come back through
// shared memory as [product][atom], two of them in turn, and leave in runs of `at` atoms: one barrier a
// batch.
//
// Bound: HBM at 8 states, the FP64 tensor pipe and the shared-memory traffic above.  Measured on a B200
// against the kernels it replaced (register products from shared memory at up to 12 states, 4 x 4-state
// tiles above), 20 orbitals: 8 states, 2,097,152 atoms, 1.29 -> 1.01 ms (5.9 TB/s); 12 states, 110,592
// atoms, 0.189 -> 0.130 ms; 40 states, 262,144 atoms, 3.53 -> 2.04 ms.  Fragments loaded straight from HBM,
// five steps ahead: 1.50, 0.196 and 2.13 ms.
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
    int at, at_log2;            // atoms a batch: a power of two, at least warps / warps_per_atom
    int stages;                 // batches in shared memory
    int state_pitch;            // elements between the states of a staged batch
    int n_used;
    int state[8 * MAX_BLOCKS];  // coefficient row of each used state, ascending
};

// Elements between the states of a staged batch: at n_orb, 64 bytes off a multiple of 128.
inline int state_pitch(int at, int n_orb) {
    const int e = at * n_orb;
    return e + (12 - e % 8) % 8;
}
template <typename RT>
size_t pair_mma_smem(int nb, int n_used, int pitch, int np, int at, int stages) {
    const int tiles = nb * (nb + 1) / 2;
    return sizeof(cx<double>) * (size_t)stages * n_used * pitch + 2 * sizeof(cx<RT>) * (size_t)np * (at + 1) +
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

// Tiles [H * TH, ...) of one atom: c is the lane's first orbital of state row 0 of block 0 (staged).
template <int NB, int WPA, int H, bool FOLD, typename RT>
__device__ __forceinline__ void atom_tiles(const cx<double>* c, int block_pitch, int n_orb, int tig, unsigned have,
                                           const short* row, int lane, cx<RT>* out, int out_pitch) {
    constexpr int T = NB * (NB + 1) / 2, TH = (T + WPA - 1) / WPA, T0 = H * TH, T1 = T0 + TH < T ? T0 + TH : T,
                  N = T1 - T0;
    double re[N][2], im[N][2];
#pragma unroll
    for (int t = 0; t < N; ++t) re[t][0] = re[t][1] = im[t][0] = im[t][1] = 0.0;
#pragma unroll 2
    for (int o = 0; o < n_orb; o += 4) {
        cx<double> v[NB];
#pragma unroll
        for (int b = 0; b < NB; ++b)
            v[b] = (o + tig < n_orb && ((have >> b) & 1u)) ? c[(size_t)b * block_pitch + o] : mk(0.0, 0.0);
#pragma unroll
        for (int t = 0; t < N; ++t) {
            const int bi = tile_row(T0 + t), bj = tile_col(T0 + t);
            mma_f64(re[t], v[bi].re, v[bj].re);
            mma_f64(im[t], v[bi].re, v[bj].im);
        }
#pragma unroll
        for (int t = 0; t < N; ++t) {
            const int bi = tile_row(T0 + t), bj = tile_col(T0 + t);
            mma_f64(re[t], v[bi].im, v[bj].im);
            if (!FOLD || bi != bj) mma_f64(im[t], -v[bi].im, v[bj].re);
        }
    }
#pragma unroll
    for (int t = 0; t < N; ++t) {
        if (FOLD && tile_row(T0 + t) == tile_col(T0 + t)) {
            // X R^T of a diagonal tile is the transpose of its R X^T: element (j, i) is held by lane 4 j +
            // i / 2 as its (i mod 2)-th
            double turned[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int from = 4 * (2 * tig + h) + (lane >> 3);
                const double e0 = __shfl_sync(0xffffffffu, im[t][0], from), e1 = __shfl_sync(0xffffffffu, im[t][1], from);
                turned[h] = (lane >> 2) & 1 ? e1 : e0;
            }
            im[t][0] -= turned[0];
            im[t][1] -= turned[1];
        }
        const short2 r = *reinterpret_cast<const short2*>(row + ((T0 + t) * 32 + lane) * 2);
        if (r.x >= 0) out[r.x * out_pitch] = narrow<RT>(mk(re[t][0], im[t][0]));
        if (r.y >= 0) out[r.y * out_pitch] = narrow<RT>(mk(re[t][1], im[t][1]));
    }
}

template <int NB, bool FOLD, typename RT>
__global__ void __launch_bounds__(32 * warps(NB), min_blocks(NB))
    k_pair_mma(const PairMmaArgs g, cx<RT>* __restrict__ rho) {
    constexpr int T = NB * (NB + 1) / 2, WARPS = warps(NB), THREADS = 32 * WARPS, WPA = warps_per_atom(NB), S = 8 * NB;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cx<double>* in = reinterpret_cast<cx<double>*>(smem_raw);  // [stages][state][state_pitch]
    const int in_stage = g.n_used * g.state_pitch;
    cx<RT>* out = reinterpret_cast<cx<RT>*>(in + (size_t)g.stages * in_stage);  // [2][product][at + 1]
    const int pitch = g.at + 1;
    short* row = reinterpret_cast<short*>(out + (size_t)2 * g.np * pitch);  // [tile][lane][2]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int grp = lane >> 2, tig = lane & 3;
    const long long batches = (g.n + g.at - 1) / g.at;
    const auto copy_in = [&](long long b, int stage) {
        if (b < batches) {
            const long long a0 = b * g.at;
            const int len = (int)min((long long)g.at, g.n - a0) * g.n_orb;
            for (int s = warp; s < g.n_used; s += WARPS) {
                const cx<double>* src = g.coeff + ((long long)g.state[s] * g.n + a0) * g.n_orb;
                cx<double>* dst = in + (size_t)stage * in_stage + (size_t)s * g.state_pitch;
                for (int e = lane; e < len; e += 32) pd_cp_async16(dst + e, src + e);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    long long b = blockIdx.x;
    for (int s = 0; s < g.stages - 1; ++s) copy_in(b + (long long)s * gridDim.x, s);
    for (int e = threadIdx.x; e < T * 64; e += THREADS) {
        const int t = e / 64, l = e / 2 % 32, h = e % 2;
        int bi = 0;
        while ((bi + 1) * (bi + 2) / 2 <= t) ++bi;
        const int bj = t - bi * (bi + 1) / 2;
        const int i = 8 * bi + l / 4, j = 8 * bj + 2 * (l % 4) + h;
        row[e] = (short)(i >= j ? g.prod[i * S + j] : -1);
    }
    unsigned have = 0;  // blocks in which this lane's state exists
#pragma unroll
    for (int k = 0; k < NB; ++k)
        if (8 * k + grp < g.n_used) have |= 1u << k;
    int stage = 0, turn = 0;
    for (; b < batches; b += gridDim.x) {
        // batch b has landed (all but the newest stages - 2 groups of this thread), everyone's copies are
        // visible, and everyone is done with the previous batch: its stage takes the next copy, and the
        // out buffer of two batches ago has been stored
        if (g.stages == 2)
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        else if (g.stages == 3)
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        else
            asm volatile("cp.async.wait_group 2;\n" ::: "memory");
        __syncthreads();
        if (turn > 0) {  // the previous batch's products
            const long long a0 = (b - gridDim.x) * g.at;
            const cx<RT>* o = out + (size_t)((turn - 1) & 1) * g.np * pitch;
            for (int e = threadIdx.x; e < g.np * g.at; e += THREADS) {
                const int p = e >> g.at_log2, k = e & (g.at - 1);
                rho[(long long)p * g.n + a0 + k] = o[p * pitch + k];  // a whole batch: not the last one
            }
        }
        const int free_stage = stage == 0 ? g.stages - 1 : stage - 1;
        copy_in(b + (long long)(g.stages - 1) * gridDim.x, free_stage);
        const cx<double>* st = in + (size_t)stage * in_stage;
        cx<RT>* o = out + (size_t)(turn & 1) * g.np * pitch;
#pragma unroll 1
        for (int a = warp / WPA; a < g.at; a += WARPS / WPA) {
            const cx<double>* c = st + (size_t)grp * g.state_pitch + a * g.n_orb + tig;
            const int bp = 8 * g.state_pitch;
            if constexpr (WPA == 1) {
                atom_tiles<NB, 1, 0, FOLD, RT>(c, bp, g.n_orb, tig, have, row, lane, o + a, pitch);
            } else {
                switch (warp % WPA) {
                    case 0: atom_tiles<NB, WPA, 0, FOLD, RT>(c, bp, g.n_orb, tig, have, row, lane, o + a, pitch); break;
                    case 1: atom_tiles<NB, WPA, 1, FOLD, RT>(c, bp, g.n_orb, tig, have, row, lane, o + a, pitch); break;
                    case 2: atom_tiles<NB, WPA, 2, FOLD, RT>(c, bp, g.n_orb, tig, have, row, lane, o + a, pitch); break;
                    default: atom_tiles<NB, WPA, 3, FOLD, RT>(c, bp, g.n_orb, tig, have, row, lane, o + a, pitch); break;
                }
            }
        }
        stage = stage + 1 == g.stages ? 0 : stage + 1;
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
