// FP64 tensor-core Gram over atoms, for every reduction that is summed in FP64: the FP64 forms, the FP32
// forms' small boxes and FP64 potentials.
//
// The reductions of CoulombCalculator::calculate (CoulombCalculator.cpp:165-172) restricted to
// atom cells and batched over the (left, right) pairs of a request, as in gram_tc.cuh:
//   C = A . B^T,  A rows = {Re V_l, Im V_l},  B rows = {Re rho_r, Im rho_r},  K = atoms,
// with FP64 products and FP64 sums on the FP64 tensor cores (mma.sync m8n8k4 .f64): FP32 operands are
// widened exactly, so the only rounding is that of FP64 accumulation.
//
// A block takes one tile of the Gram (gram_blocks.hpp) and an atom range, in chunks of KC atoms (32, or 64
// where the warps split the atoms and the box has enough of them, so that a chunk's barrier and copies
// are spread over more MMAs):
//   copy      cp.async of the chunk's raw complex values, 1 to 3 chunks ahead ([density][KC + 4], 16
//             bytes a copy, 8 for FP32 rows that do not start on a 16-byte boundary);
//   multiply  8 warps as WR x WC x KS: warp (wr, wc, ks) holds the 8 x 8 tiles (wr + WR a, wc + WC b) of
//             C, a < A, b < B, over every KS-th k-step of 4 atoms.  A fragment value is one shared load
//             (re or im of an operand value; the pitch of KC + 4 puts a warp's 32 on distinct banks) and,
//             for FP32 operands, one conversion.
// At the end the KS partial sums are added through shared memory and the results go to out4 with FP64
// atomics.  Every MMA of the A x B register tile is issued whether its rows exist or not (a predicated-off
// one takes its 16 pipe cycles all the same), so the host picks A, B and the warp grid to fit: splitting
// the warps over atoms keeps them at full register tiles (20 densities a side: 5 x 5 tiles, which a
// 2 x 4 grid of 3 x 2 would fill to 52 %).
//
// Bound: the FP64 tensor pipe (64 FMA a clock and SM measured, 18.2 T FMA/s) at many densities, the
// latency of the chunks of a small box at few.  Measured on a B200 against the kernels this one replaced
// (register products for FP64 operands; every pair of densities, FP32 operands widened into a second
// stage, a 2 x 4 warp grid for any tile): 96^3 box, 12 states in FP64 (42 and 36 densities, 6 symmetric
// tiles) 0.898 -> 0.186 ms, the FP64 tensor pipe half busy; six boxes of 13,824 to 24,192 atoms, 8
// states, FP32: 0.346 -> 0.144 ms; 64^3 grid product 0.085 -> 0.027 ms; 4,096 atoms, 4 states,
// 18.9 -> 10.0 us.
#pragma once

#include <cstdint>

#include "fft.cuh"
#include "gram_blocks.hpp"

namespace clk {
namespace dm {

__host__ __device__ constexpr int pitch(int kc) { return kc + 4; }  // complex elements per staged density
constexpr int WARPS = 8;
constexpr int THREADS = 32 * WARPS;
constexpr int WIDTH = 64;      // densities a tile side, at most

template <typename S>
struct GramArgs {
    const cx<S>* V;       // left densities: V[(lidx ? lidx[l] : l) * v_stride + atom]
    const int* lidx;
    long long v_stride;
    const int* ridx;      // right densities: rho[(ridx ? ridx[r] : r) * r_stride + atom]
    long long r_stride;
    long long na;               // atoms
    long long atoms_per_split;  // a multiple of the chunk
    int stages;                 // chunks in shared memory
    int nd_a, nd_b;             // staged densities of the largest tile, a side (multiples of 4)
    int wr, wc;                 // warp grid over the C tile; 8 / (wr * wc) k slices
    int align_v, align_r;       // every row of the operand starts on a 16-byte boundary
    double* out4;               // out4[l][r] += {ac, bd, ad, bc}
    GramTiles tiles;
};

template <typename SV, typename SR>
__host__ __device__ constexpr size_t stage_bytes(int kc, int nd_a, int nd_b) {
    return (size_t)pitch(kc) * (nd_a * sizeof(cx<SV>) + nd_b * sizeof(cx<SR>));
}
// Shared memory of the reduction over k slices: half the slices' sums at a time.
__host__ __device__ constexpr size_t reduce_bytes(int a, int b, int slices) {
    return slices > 1 ? (size_t)(WARPS / 2) * a * b * 2 * 32 * sizeof(double) : 0;
}

__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}
template <int BYTES>
__device__ __forceinline__ void cp_async_part(void* dst, const void* src, unsigned bytes) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

// Copies atoms [k0, k0 + KC) of n densities (rows beyond n, up to n4, and atoms beyond k_end as zeros).
template <int KC, typename S, typename ROW>
__device__ __forceinline__ void copy_chunk(cx<S>* dst, int n, int n4, long long k0, long long k_end, bool aligned,
                                           const cx<S>* any, ROW&& row) {
    constexpr int PITCH = pitch(KC), PER = 16 / sizeof(cx<S>);  // PER: atoms per 16-byte copy
    if (aligned) {
        for (int e = threadIdx.x; e < n4 * (KC / PER); e += THREADS) {
            const int i = e / (KC / PER), k = (e % (KC / PER)) * PER;
            const long long left = i < n ? k_end - (k0 + k) : 0;
            const unsigned bytes = left >= PER ? 16u : left > 0 ? (unsigned)(left * sizeof(cx<S>)) : 0u;
            cp_async_part<16>(dst + i * PITCH + k, bytes ? row(i) + k0 + k : any, bytes);
        }
    } else {
        for (int e = threadIdx.x; e < n4 * KC; e += THREADS) {
            const int i = e / KC, k = e % KC;
            const bool in = i < n && k0 + k < k_end;
            if constexpr (sizeof(cx<S>) == 16)
                cp_async_part<16>(dst + i * PITCH + k, in ? row(i) + k0 + k : any, in ? 16u : 0u);
            else
                cp_async_part<8>(dst + i * PITCH + k, in ? row(i) + k0 + k : any, in ? 8u : 0u);
        }
    }
}

template <typename SV, typename SR, int KC, int A, int B>
__global__ void __launch_bounds__(THREADS, 1) k_gram_dmma(const cx<SR>* __restrict__ rho, const GramArgs<SV> g) {
    constexpr int PITCH = pitch(KC);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int left_row[WIDTH], right_row[WIDTH];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    GramTile tile;
    gram_tile(g.tiles, blockIdx.x, &tile);
    const int nA4 = (tile.nl + 3) & ~3, nB4 = (tile.nr + 3) & ~3;
    const int ta = nA4 / 4, tb = nB4 / 4;  // 8-row tiles of C
    const long long k_begin = (long long)blockIdx.y * g.atoms_per_split;
    const long long k_end = min(g.na, k_begin + g.atoms_per_split);
    const int nc = (int)((k_end - k_begin + KC - 1) / KC);
    const size_t stage = stage_bytes<SV, SR>(KC, g.nd_a, g.nd_b);
    const size_t b_off = (size_t)PITCH * g.nd_a * sizeof(cx<SV>);
    for (int r = threadIdx.x; r < tile.nr; r += THREADS)
        right_row[r] = g.ridx ? g.ridx[tile.r0 + r] : tile.r0 + r;
    for (int l = threadIdx.x; l < tile.nl; l += THREADS)
        left_row[l] = g.lidx ? g.lidx[tile.l0 + l] : tile.l0 + l;
    __syncthreads();
    const auto issue = [&](int c) {
        unsigned char* st = smem_raw + (size_t)(c % g.stages) * stage;
        const long long k0 = k_begin + (long long)c * KC;
        copy_chunk<KC, SV>(reinterpret_cast<cx<SV>*>(st), tile.nl, nA4, k0, k_end, g.align_v, g.V,
                       [&](int i) { return g.V + (long long)left_row[i] * g.v_stride; });
        copy_chunk<KC, SR>(reinterpret_cast<cx<SR>*>(st + b_off), tile.nr, nB4, k0, k_end, g.align_r, rho,
                       [&](int i) { return rho + (long long)right_row[i] * g.r_stride; });
    };
    const int slices = WARPS / (g.wr * g.wc);
    const int ks0 = warp % slices, wr = warp / slices % g.wr, wc = warp / slices / g.wr;
    const int grp = lane >> 2, tig = lane & 3;
    double acc[A][B][2];
#pragma unroll
    for (int a = 0; a < A; ++a)
#pragma unroll
        for (int b = 0; b < B; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
    for (int c = 0; c < g.stages - 1; ++c) {
        if (c < nc) issue(c);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
#pragma unroll 1
    for (int c = 0; c < nc; ++c) {
        // chunk c has landed: all but the newest stages - 2 groups of this thread are complete
        if (g.stages == 4)
            asm volatile("cp.async.wait_group 2;" ::: "memory");
        else if (g.stages == 3)
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        else
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // everyone's copies of chunk c, and everyone is done with chunk c - 1
        if (c + g.stages - 1 < nc) issue(c + g.stages - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const unsigned char* st = smem_raw + (size_t)(c % g.stages) * stage;
        const SV* sa = reinterpret_cast<const SV*>(st) + (size_t)(grp >> 1) * (2 * PITCH) + (grp & 1);
        const SR* sb = reinterpret_cast<const SR*>(st + b_off) + (size_t)(grp >> 1) * (2 * PITCH) + (grp & 1);
#pragma unroll 2
        for (int ks = ks0; ks < KC / 4; ks += slices) {
            const int k = 2 * (ks * 4 + tig);
            double af[A], bf[B];
#pragma unroll
            for (int a = 0; a < A; ++a) {
                const int ti = wr + g.wr * a;
                af[a] = ti < ta ? (double)sa[ti * (8 * PITCH) + k] : 0.0;
            }
#pragma unroll
            for (int b = 0; b < B; ++b) {
                const int tj = wc + g.wc * b;
                bf[b] = tj < tb ? (double)sb[tj * (8 * PITCH) + k] : 0.0;
            }
#pragma unroll
            for (int a = 0; a < A; ++a)
#pragma unroll
                for (int b = 0; b < B; ++b) mma_f64(acc[a][b], af[a], bf[b]);
        }
    }
    // the k slices' sums: the upper half of the slices hands its sums to the lower half, until one is left
    double* red = reinterpret_cast<double*>(smem_raw);
#pragma unroll 1
    for (int h = slices / 2; h >= 1; h /= 2) {
        double* mine = red + (size_t)((warp / slices) * h + (ks0 & (h - 1))) * (A * B * 2 * 32) + lane;
        __syncthreads();
        if (ks0 >= h && ks0 < 2 * h) {
#pragma unroll
            for (int a = 0; a < A; ++a)
#pragma unroll
                for (int b = 0; b < B; ++b) {
                    mine[(a * B + b) * 64] = acc[a][b][0];
                    mine[(a * B + b) * 64 + 32] = acc[a][b][1];
                }
        }
        __syncthreads();
        if (ks0 < h) {
#pragma unroll
            for (int a = 0; a < A; ++a)
#pragma unroll
                for (int b = 0; b < B; ++b) {
                    acc[a][b][0] += mine[(a * B + b) * 64];
                    acc[a][b][1] += mine[(a * B + b) * 64 + 32];
                }
        }
    }
    if (ks0 != 0) return;
#pragma unroll
    for (int a = 0; a < A; ++a)
#pragma unroll
        for (int b = 0; b < B; ++b) {
            const int ti = wr + g.wr * a, tj = wc + g.wc * b;
            const int row = ti * 8 + grp, l = row >> 1, pa = row & 1;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int col = tj * 8 + 2 * tig + h, r = col >> 1, pc = col & 1;
                if (l < tile.nl && r < tile.nr && l + tile.diag >= r) {
                    const int qi = (pa == pc) ? pa : 2 + pa;  // ac, bd, ad, bc
                    atomicAdd(g.out4 + ((long long)(tile.l0 + l) * g.tiles.ldr + tile.r0 + r) * 4 + qi, acc[a][b][h]);
                }
            }
        }
}

}  // namespace dm
}  // namespace clk
