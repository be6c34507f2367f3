// Split-precision tensor-core Gram over atoms (FP32 form).
//
// The reductions of CoulombCalculator::calculate (CoulombCalculator.cpp:165-172), restricted
// to atom cells and batched over every (left, right) pair of a request, form the real Gram
//   C = A . B^T,  A rows = {Re V_l, Im V_l} (2 per left density),
//                 B rows = {Re rho_r, Im rho_r} (2 per right density),  K = atoms,
// whose 2x2 blocks are {sum ac, sum ad; sum bc, sum bd} for V = a+ib, rho = c+id.
//
// Each FP64 operand is split into two TF32 parts, x = hi + lo (both rounded to nearest), and
// C = A_hi.B_hi + (A_hi.B_lo + A_lo.B_hi) is accumulated by tcgen05 MMAs (kind::tf32, M=128,
// N=128, K=8) in FP32 in tensor memory.  The tensor cores' FP32 accumulation rounds toward
// zero, a bias that grows with every MMA added into a running sum.  So the main products go to
// an accumulator that is drained into FP64 registers after every k-tile of 32 atoms (4 MMAs,
// double-buffered in tensor memory), while the two correction products -- 2^-11 of the main
// ones and of random sign, the lo parts being round-to-nearest residuals -- accumulate in a
// third accumulator over the block's whole atom range and are drained once.  The drained
// partial sums are added across the atom range in FP64 and then across atom splits with FP64
// atomics.  The dropped lo.lo term and
// the rounding of the parts are ~2^-22 of each product.
//
// Operands are staged by TMA (no multicast) into 128-byte-swizzled shared-memory tiles: one
// warp issues the copies, one lane issues the MMAs, sixteen warps drain the accumulator.
// Every wait is bounded by a clock deadline; on expiry the block records an error in the
// slot after the results, waits (again bounded) for its own copies and MMAs, frees its
// tensor memory and returns.
#pragma once

#include <cuda.h>
#include <cstdint>

#include "fft.cuh"
#include "gram_blocks.hpp"

namespace clk {
namespace tc {

constexpr int BM = 128;          // A rows per tile (64 left densities)
constexpr int BN = 128;          // B rows per tile (64 right densities)
constexpr int BK = 32;           // atoms per k-tile: 32 x 4 B = one 128-byte swizzle row
constexpr int STAGES = 3;        // shared-memory pipeline depth
constexpr int CH = 1;            // k-tiles per FP32 accumulation chunk (32 atoms)
constexpr int A_BYTES = BM * BK * 4;
constexpr int B_BYTES = BN * BK * 4;
constexpr int STAGE_BYTES = 2 * A_BYTES + 2 * B_BYTES;  // hi and lo of both operands
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
// Sixteen warps hide each other's tensor-memory waits: the 40-state Gram took 6.03 ms with eight.  What is
// left per k-tile (1.10 us) is near the 64 KB of operands each SM draws from L2 (8.8 TB/s over all SMs).
constexpr int EPI_WARPS = 16;
constexpr int EPI_COLS = 4 * BN / EPI_WARPS;  // accumulator columns a warp drains (of its 32 lanes)
constexpr int THREADS = 32 * (2 + EPI_WARPS);
constexpr uint32_t TMEM_COLS = 4 * BN;  // main x double buffer, correction, unused; FP32
constexpr long long TIMEOUT_CYCLES = 1LL << 32;  // ~2 s at B200 clocks

static_assert(BN == 128 && BM == 128, "epilogue mapping assumes 128x128 tiles");

// Instruction descriptor, kind::tf32: D F32 (bits 4-5 = 1), A and B TF32 (bits 7-9, 10-12
// = 2), both K-major (bits 15, 16 = 0), N >> 3 at bit 17, M >> 4 at bit 24.
constexpr uint32_t IDESC = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(BN >> 3) << 17) |
                           ((uint32_t)(BM >> 4) << 24);

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t a, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t a, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(a), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t a) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(a) : "memory");
}
__device__ __forceinline__ bool mbar_test(uint32_t a, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    return ok != 0;
}
// Waits for the phase of parity `parity` to complete.  Returns false when the deadline
// passes (and raises the block's abort flag) or when another role has already aborted.
__device__ __forceinline__ bool mbar_wait(uint32_t a, uint32_t parity, volatile int* abort_flag) {
    const long long t0 = clock64();
    while (!mbar_test(a, parity)) {
        if (*abort_flag) return false;
        if (clock64() - t0 > TIMEOUT_CYCLES) {
            *abort_flag = 1;
            return false;
        }
    }
    return true;
}
// Teardown wait that ignores the abort flag (still bounded).
__device__ __forceinline__ void mbar_drain(uint32_t a, uint32_t parity) {
    const long long t0 = clock64();
    while (!mbar_test(a, parity))
        if (clock64() - t0 > TIMEOUT_CYCLES) return;
}

// Tile (x = atom, y = row, z = part) of a [part][row][atom] operand; rows beyond the operand's
// real rows are filled with zeros by the copy itself (nothing is read for them).
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z,
                                            uint32_t mbar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(mbar)
        : "memory");
}

// Shared-memory matrix descriptor of a K-major tile with the 128-byte swizzle: start address
// >> 4, leading offset 1 (unused for swizzled K-major), stride 1024 B between 8-row groups,
// descriptor version 1 (bit 46), layout type 2 = SWIZZLE_128B (bits 61-63).
__device__ __forceinline__ uint64_t sw128_desc(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) |
           (2ull << 61);
}

__device__ __forceinline__ void mma_tf32(uint32_t d, uint64_t a, uint64_t b, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(IDESC), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Issues the load of 8 consecutive FP32 accumulator columns of this thread's lane (no wait).
__device__ __forceinline__ void tmem_ld8_issue(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
// Waits for this thread's tensor-memory loads; the 16 destination registers pass through the
// wait, so that no use of them is scheduled before it.
__device__ __forceinline__ void tmem_wait_ld16(uint32_t* r) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                   "+r"(r[15])
                 :
                 : "memory");
}

__device__ __forceinline__ float tf32_rn(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
}

// ---------------------------------------------------------------------------------------
// Split pass: density d of `src` (row idx[d], or d; complex of S) over atoms [a0, a0 + na) ->
//   dst[part][2d + {0: re, 1: im}][k], part 0 = hi, 1 = lo, 2n rows a part; k >= na are zero.
// grid.y = n densities, grid.x strides over k.  (The Gram's tiles are 128 rows; its copies fill
// the rows beyond 2n with zeros, so no padding is stored.)
// ---------------------------------------------------------------------------------------
template <typename S>
__global__ void __launch_bounds__(256) k_tf32_split(const cx<S>* __restrict__ src, long long stride,
                                                    const int* __restrict__ idx, int n, long long a0,
                                                    long long na, long long k_pad, float* __restrict__ dst) {
    const int d = blockIdx.y;
    const long long plane = (long long)(2 * n) * k_pad;
    float* hre = dst + (long long)(2 * d) * k_pad;
    float* him = hre + k_pad;
    const cx<S>* s = src + (long long)(idx ? idx[d] : d) * stride + a0;
    for (long long k = blockIdx.x * 256LL + threadIdx.x; k < k_pad; k += (long long)gridDim.x * 256) {
        double re = 0.0, im = 0.0;
        if (k < na) {
            const cx<S> z = s[k];
            re = (double)z.re;
            im = (double)z.im;
        }
        const float hr = tf32_rn((float)re), hi_ = tf32_rn((float)im);
        hre[k] = hr;
        him[k] = hi_;
        hre[plane + k] = tf32_rn((float)(re - (double)hr));
        him[plane + k] = tf32_rn((float)(im - (double)hi_));
    }
}

// ---------------------------------------------------------------------------------------
// The Gram.  grid = (tiles, splits), tiles of at most 64 x 64 densities (gram_blocks.hpp); split y covers
// k-tiles [y * kt_per, min(kt_total, (y + 1) * kt_per)), never empty.  out4[l][r] += {ac, bd, ad, bc};
// *err (as int) is set to 1 if any wait expired.
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(THREADS, 1)
    k_gram_tc(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, int kt_total,
              int kt_per, const GramTiles tiles, double* __restrict__ out4, double* __restrict__ err) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* gbase = smem_raw + (base - raw);
    uint64_t* bars = reinterpret_cast<uint64_t*>(gbase + STAGES * STAGE_BYTES);
    // bars: full[STAGES], empty[STAGES], acc_full[2], acc_empty[2], drain
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 5);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const auto bar = [&](int i) { return smem_u32(bars + i); };
    const int FULL = 0, EMPTY = STAGES, ACCF = 2 * STAGES, ACCE = 2 * STAGES + 2, DRAIN = 2 * STAGES + 4;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    GramTile tile;
    gram_tile(tiles, blockIdx.x, &tile);
    const int m0 = 2 * tile.l0, n0 = 2 * tile.r0;
    const int kt0 = blockIdx.y * kt_per;
    const int kt1 = min(kt_total, kt0 + kt_per);
    const int nchunks = (kt1 - kt0 + CH - 1) / CH;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(bar(FULL + s), 1);
            mbar_init(bar(EMPTY + s), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(bar(ACCF + b), 1);
            mbar_init(bar(ACCE + b), EPI_WARPS);  // one arrival a warp, after __syncwarp
        }
        mbar_init(bar(DRAIN), 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            // ---- TMA producer ----
            int s = 0;
            uint32_t ph = 0;
            int issued = 0;
            for (int kt = kt0; kt < kt1; ++kt) {
                if (!mbar_wait(bar(EMPTY + s), ph ^ 1u, abort_flag)) break;
                const uint32_t st = base + (uint32_t)(s * STAGE_BYTES);
                mbar_expect_tx(bar(FULL + s), STAGE_BYTES);
                const int x = kt * BK;
                tma_load_3d(st, &mapA, x, m0, 0, bar(FULL + s));
                tma_load_3d(st + A_BYTES, &mapA, x, m0, 1, bar(FULL + s));
                tma_load_3d(st + 2 * A_BYTES, &mapB, x, n0, 0, bar(FULL + s));
                tma_load_3d(st + 2 * A_BYTES + B_BYTES, &mapB, x, n0, 1, bar(FULL + s));
                ++issued;
                if (++s == STAGES) {
                    s = 0;
                    ph ^= 1u;
                }
            }
            if (*abort_flag) {
                // let the last (up to STAGES) copies land before the block's memory goes away
                for (int i = 1; i <= min(issued, STAGES); ++i) {
                    const int n = issued - i;
                    mbar_drain(bar(FULL + n % STAGES), (uint32_t)((n / STAGES) & 1));
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // ---- MMA issuer ----
            int s = 0;
            uint32_t ph = 0;
            int kt = kt0;
            bool issued_any = false;
            for (int ch = 0; ch < nchunks; ++ch) {
                const int b = ch & 1;
                if (!mbar_wait(bar(ACCE + b), (uint32_t)(((ch >> 1) & 1) ^ 1), abort_flag)) break;
                fence_after();
                const uint32_t dm = tmem + (uint32_t)(b * BN);  // main products of this chunk
                const uint32_t dc = tmem + (uint32_t)(2 * BN);  // correction products, whole range
                const int kend = min(kt1, kt + CH);
                bool ok = true;
                uint32_t acc = 0;
                for (; kt < kend; ++kt) {
                    if (!mbar_wait(bar(FULL + s), ph, abort_flag)) {
                        ok = false;
                        break;
                    }
                    fence_after();
                    const uint32_t st = base + (uint32_t)(s * STAGE_BYTES);
#pragma unroll
                    for (int kk = 0; kk < BK / 8; ++kk) {
                        const uint64_t ahi = sw128_desc(st + kk * 32);
                        const uint64_t alo = sw128_desc(st + A_BYTES + kk * 32);
                        const uint64_t bhi = sw128_desc(st + 2 * A_BYTES + kk * 32);
                        const uint64_t blo = sw128_desc(st + 2 * A_BYTES + B_BYTES + kk * 32);
                        mma_tf32(dm, ahi, bhi, acc);
                        mma_tf32(dc, alo, bhi, (ch > 0 || acc) ? 1u : 0u);
                        mma_tf32(dc, ahi, blo, 1u);
                        acc = 1u;
                    }
                    issued_any = true;
                    mma_commit(bar(EMPTY + s));  // the stage is free once these MMAs finish
                    if (++s == STAGES) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
                if (!ok) break;
                mma_commit(bar(ACCF + b));  // chunk complete in accumulator b
            }
            if (*abort_flag && issued_any) {
                mma_commit(bar(DRAIN));
                mbar_drain(bar(DRAIN), 0);
            }
        }
    } else {
        // ---- epilogue: FP32 accumulator -> FP64 registers ----
        const int q = warp & 3;                      // tensor-memory lane quarter this warp may read
        const int c0 = ((warp - 2) >> 2) * EPI_COLS;  // first of its columns
        double acc[EPI_COLS];
#pragma unroll
        for (int i = 0; i < EPI_COLS; ++i) acc[i] = 0.0;
        const uint32_t lanes = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)c0;
        const auto drain = [&](uint32_t col) {
#pragma unroll
            for (int j = 0; j < EPI_COLS / 16; ++j) {
                uint32_t v[16];
                tmem_ld8_issue(lanes + col + 16 * j, v);
                tmem_ld8_issue(lanes + col + 16 * j + 8, v + 8);
                tmem_wait_ld16(v);
#pragma unroll
                for (int i = 0; i < 16; ++i) acc[16 * j + i] += (double)__uint_as_float(v[i]);
            }
        };
        bool ok = true;
        for (int ch = 0; ch < nchunks; ++ch) {
            const int b = ch & 1;
            bool got = mbar_wait(bar(ACCF + b), (uint32_t)((ch >> 1) & 1), abort_flag);
            got = __all_sync(0xffffffffu, got);
            if (!got) {
                ok = false;
                break;
            }
            fence_after();
            drain((uint32_t)(b * BN));
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(ACCE + b));
        }
        if (ok) {
            // the correction accumulator is complete with the last chunk's commit
            fence_after();
            drain((uint32_t)(2 * BN));
            const int R = 32 * q + lane;
            const int l = R >> 1, pa = R & 1;
            if (l < tile.nl) {
                double* row = out4 + ((long long)(tile.l0 + l) * tiles.ldr + tile.r0) * 4;
#pragma unroll
                for (int j = 0; j < EPI_COLS; ++j) {
                    const int Cg = c0 + j;
                    const int r = Cg >> 1, pc = Cg & 1;
                    if (r < tile.nr) {
                        const int qi = (pa == pc) ? pa : 2 + pa;  // ac, bd, ad, bc
                        atomicAdd(row + 4 * r + qi, acc[j]);
                    }
                }
            }
        }
    }

    fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag)
        *reinterpret_cast<volatile int*>(err) = 1;
    if (warp == 1) {
        __syncwarp();
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

// ---------------------------------------------------------------------------------------
// Fused Gram for FP32 operands (the FP32 sub-lattice form: FP32 potentials and pair densities).
// The split happens inside the kernel, so neither the hi/lo operands nor any padding reach HBM: raw complex
// values come by cp.async into a ring of AHEAD + 1 slots, and their TF32 parts go with four 16-byte stores (re hi, im
// hi, re lo, im lo of 4 atoms) into the MMA stage in the 128-byte-swizzled K-major layout the descriptors expect --
// row r, atoms 4c..4c+3 at (r/8)*1024 + (r%8)*128 + ((c ^ (r%8))*16): 8 lanes fill one row without bank
// conflicts.  The MMAs' N is the block's right rows rounded up to 16.  Rows beyond the real ones are zeroed once at
// the start and never written again.
// ---------------------------------------------------------------------------------------
struct FusedGram {
    const float2* V;      // left densities: V[(lidx ? lidx[l] : l) * v_stride + atom]
    const int* lidx;
    long long v_stride;
    const float2* rho;    // right densities: rho[(ridx ? ridx[r] : r) * r_stride + atom]
    long long r_stride;
    const int* ridx;
    long long na;         // atoms
    int kt_total, kt_per;
    uint32_t stage_bytes;     // 2 * BM * 128 + 2 * nb_max * 128
    uint32_t raw_slot_bytes;  // (left + right densities of a block, at most) * 32 * 8
    double* out4;
    double* err;
    int aligned16;            // every density row starts on a 16-byte boundary (16-byte copies)
    GramTiles tiles;
};

constexpr int FUSED_MAX_DENS = BM / 2 + BN / 2;  // densities a block converts per k-tile

__host__ __device__ constexpr uint32_t fused_idesc(int nb) {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(nb >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}
// Byte offset of the 16-byte chunk c (atoms 4c..4c+3) of row r in a 128-byte-swizzled tile.
__device__ __forceinline__ uint32_t sw128_chunk(int row, int c) {
    return (uint32_t)((row >> 3) * 1024 + (row & 7) * 128 + ((c ^ (row & 7)) << 4));
}
__device__ __forceinline__ void mma_tf32_n(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src, uint32_t src_bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
// 16 bytes, of which the first src_bytes (0, 8 or 16) are read and the rest zero-filled.
__device__ __forceinline__ void cp_async16z(uint32_t dst, const void* src, uint32_t src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ---------------------------------------------------------------------------------------
// The fused Gram with its roles in separate warps (at most 48 right densities a block: N <= 96),
// so that the conversion of k-tile t + 1, the MMAs of k-tile t and the drain of k-tile t - 1
// run at the same time instead of one after another in every warp:
//   warps 0-6    copy their items' raw values AHEAD k-tiles ahead with cp.async (16 bytes on
//                rows that start on a 16-byte boundary, else 8; each thread reads back only its
//                own copies) and convert them: item (density i, atoms 4q .. 4q + 3) -> TF32 hi
//                and lo of re and im, four 16-byte stores into the 128-byte-swizzled K-major
//                stage; then one arrival a warp on the stage's full barrier;
//   warp 7       lane 0 issues the tile's 12 MMAs once the stage is full and its accumulator
//                buffer drained (three main buffers in tensor memory, the correction in a
//                fourth), and commits them to the stage's empty and the buffer's full barrier;
//   warps 8-     drain: 8 of them up to N = 80, 12 above (36 densities a side: 0.472 ms with 8, 0.483 with
//                12); warp w reads lane quarter w % 4 and its share (a half, a third) of the column groups
//                of 8, two k-tiles at a time, into FP64 registers.  PAIRS: the two FP32 values of a
//                column are summed once first (round to nearest, unbiased, at most 2^-24 of the pair
//                against the TF32 parts' 2^-22 of each product); only where one tile of at most 40
//                right densities holds the request.  The correction accumulator comes once, after the
//                last k-tile.
// TF32 rounding to nearest (ties away from zero, as cvt.rna.tf32.f32 for finite values) is done
// on the integer pipe: add half the weight of the 13 dropped mantissa bits, clear them.
// ---------------------------------------------------------------------------------------
constexpr int WS_CONV_WARPS = 7;
constexpr int WS_MMA_WARP = 7;
constexpr int WS_DRAIN_WARP0 = 8;
constexpr int ws_threads(int drains) { return 32 * (WS_DRAIN_WARP0 + drains); }
constexpr int WS_NACC = 3;         // main accumulator buffers (128 columns apart)
constexpr int WS_STAGES = 2;       // MMA operand stages in shared memory
constexpr int WS_MAX_NB = 96;      // MMA N: at most 48 right densities
constexpr int WS_MAX_NB8 = 80;     // with 8 drain warps: at most 40
// items of 4 atoms a converter thread takes: 64 left + 40 right densities, 8 items each
constexpr int WS_ITEMS = ((BM / 2 + WS_MAX_NB / 2) * (BK / 4) + 32 * WS_CONV_WARPS - 1) / (32 * WS_CONV_WARPS);

// Bytes of dynamic shared memory: alignment slack, the MMA stages, the raw ring, the source
// table and the barriers.
__host__ __device__ constexpr size_t ws_smem_bytes(uint32_t stage_bytes, uint32_t raw_slot_bytes, int ahead) {
    return 1024 + (size_t)WS_STAGES * stage_bytes + (size_t)(ahead + 1) * raw_slot_bytes +
           sizeof(void*) * FUSED_MAX_DENS + 256;
}

__device__ __forceinline__ uint32_t tf32_rna_bits(uint32_t b) { return (b + 0x1000u) & 0xFFFFE000u; }

// 8 consecutive FP32 accumulator columns of this thread's lane.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

template <int AHEAD, int DRAINS, bool PAIRS>
__global__ void __launch_bounds__(ws_threads(DRAINS), 1) k_gram_tc_ws(const FusedGram g) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char* gbase = smem_raw + (base - raw);
    const uint32_t ring_off = WS_STAGES * g.stage_bytes;
    const float2** src_tab = reinterpret_cast<const float2**>(gbase + ring_off + (AHEAD + 1) * g.raw_slot_bytes);
    uint64_t* bars = reinterpret_cast<uint64_t*>(src_tab + FUSED_MAX_DENS);
    // bars: full[WS_STAGES], empty[WS_STAGES], acc_full[WS_NACC], acc_empty[WS_NACC], drain
    constexpr int FULL = 0, EMPTY = WS_STAGES, ACCF = 2 * WS_STAGES, ACCE = ACCF + WS_NACC, DRAIN = ACCE + WS_NACC;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + DRAIN + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const auto bar = [&](int i) { return smem_u32(bars + i); };
    constexpr uint32_t A_PART = BM * 128;
    const uint32_t b_part = (g.stage_bytes - 2u * A_PART) / 2u;
    constexpr int CONV_THREADS = 32 * WS_CONV_WARPS;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    GramTile tile;
    gram_tile(g.tiles, blockIdx.x, &tile);
    const int la0 = tile.l0, rb0 = tile.r0, nA = tile.nl, nB = tile.nr;
    const int nd = nA + nB;
    const int nb = max(16, (2 * nB + 15) / 16 * 16);
    const uint32_t idesc = fused_idesc(nb);
    const int kt0 = blockIdx.y * g.kt_per;
    const int nt = min(g.kt_total, kt0 + g.kt_per) - kt0;

    if (threadIdx.x == 0) {
        // one arrival a warp (after __syncwarp): full by the converter warps, drained by the
        // drain warps
        for (int s = 0; s < WS_STAGES; ++s) {
            mbar_init(bar(FULL + s), WS_CONV_WARPS);
            mbar_init(bar(EMPTY + s), 1);
        }
        for (int b = 0; b < WS_NACC; ++b) {
            mbar_init(bar(ACCF + b), 1);
            mbar_init(bar(ACCE + b), DRAINS);
        }
        mbar_init(bar(DRAIN), 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    constexpr int WS_THREADS = 32 * (WS_DRAIN_WARP0 + DRAINS);
    for (int i = threadIdx.x; i < nd; i += WS_THREADS) {
        if (i < nA) {
            src_tab[i] = g.V + (long long)(g.lidx ? g.lidx[la0 + i] : la0 + i) * g.v_stride;
        } else {
            const int r = rb0 + (i - nA);
            src_tab[i] = g.rho + (long long)(g.ridx ? g.ridx[r] : r) * g.r_stride;
        }
    }
    // zero both MMA stages once: rows beyond the real ones are never written again
    for (uint32_t o = threadIdx.x * 16u; o < ring_off; o += WS_THREADS * 16u)
        *reinterpret_cast<uint4*>(gbase + o) = make_uint4(0u, 0u, 0u, 0u);
    fence_proxy_async();
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;
    bool ok = true;

    if (warp < WS_CONV_WARPS) {
        // ---- converters: item it = (density it / 8, atoms 4 (it % 8) .. + 3); the raw slot holds
        // atoms 4q, 4q + 1 of item it at 16 it and atoms 4q + 2, 4q + 3 at half + 16 it, so that
        // consecutive threads copy and read contiguous 16-byte pieces.  A thread's items, their
        // sources and their places in the stage are the same for every k-tile.
        const int items = nd * (BK / 4);
        const uint32_t half = (uint32_t)items * 16u;
        const float2* isrc[WS_ITEMS];
        uint32_t ihi[WS_ITEMS][2], ilo[WS_ITEMS][2];
#pragma unroll
        for (int k = 0; k < WS_ITEMS; ++k) {
            const int it = threadIdx.x + k * CONV_THREADS;
            const int i = min(it, items - 1) >> 3, qd = it & 7;
            const bool left = i < nA;
            const int row = 2 * (left ? i : i - nA);
            const uint32_t hi0 = left ? 0u : 2u * A_PART, lo0 = hi0 + (left ? A_PART : b_part);
            isrc[k] = src_tab[i] + 4 * qd;
            ihi[k][0] = hi0 + sw128_chunk(row, qd);
            ihi[k][1] = hi0 + sw128_chunk(row + 1, qd);
            ilo[k][0] = lo0 + sw128_chunk(row, qd);
            ilo[k][1] = lo0 + sw128_chunk(row + 1, qd);
        }
        const auto issue = [&](int t) {
            const long long at0 = (long long)(kt0 + t) * BK;
            const uint32_t slot = base + ring_off + (uint32_t)(t % (AHEAD + 1)) * g.raw_slot_bytes;
#pragma unroll
            for (int k = 0; k < WS_ITEMS; ++k) {
                const int it = threadIdx.x + k * CONV_THREADS;
                if (it < items) {
                    const long long a = at0 + 4 * (it & 7);  // first atom of the item
                    const uint32_t d0 = slot + (uint32_t)it * 16u;
                    if (g.aligned16) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const long long left_atoms = g.na - (a + 2 * h);
                            const uint32_t nbytes = left_atoms >= 2 ? 16u : (left_atoms == 1 ? 8u : 0u);
                            cp_async16z(d0 + h * half, isrc[k] + (nbytes ? at0 + 2 * h : -4LL * (it & 7)), nbytes);
                        }
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const bool in = a + e < g.na;
                            cp_async8(d0 + (e >> 1) * half + 8u * (e & 1), isrc[k] + (in ? at0 + e : -4LL * (it & 7)),
                                      in ? 8u : 0u);
                        }
                    }
                }
            }
        };
#pragma unroll 1
        for (int t = 0; t < AHEAD; ++t) {
            if (t < nt) issue(t);
            cp_async_commit();
        }
#pragma unroll 1
        for (int t = 0; t < nt; ++t) {
            if (t + AHEAD < nt) issue(t + AHEAD);
            cp_async_commit();
            cp_async_wait<AHEAD>();  // this thread's copies of k-tile t have landed
            const int s = t % WS_STAGES;
            const bool got = mbar_wait(bar(EMPTY + s), (uint32_t)(((t / WS_STAGES) & 1) ^ 1), abort_flag);
            if (!__all_sync(0xffffffffu, got)) {
                ok = false;
                break;
            }
            unsigned char* stg = gbase + (size_t)s * g.stage_bytes;
            const unsigned char* rs = gbase + ring_off + (size_t)(t % (AHEAD + 1)) * g.raw_slot_bytes;
#pragma unroll
            for (int k = 0; k < WS_ITEMS; ++k) {
                const int it = threadIdx.x + k * CONV_THREADS;
                if (it < items) {
                    const uint4 z0 = *reinterpret_cast<const uint4*>(rs + it * 16);         // re0 im0 re1 im1
                    const uint4 z1 = *reinterpret_cast<const uint4*>(rs + half + it * 16);  // re2 im2 re3 im3
                    const uint32_t re[4] = {z0.x, z0.z, z1.x, z1.z}, im[4] = {z0.y, z0.w, z1.y, z1.w};
                    uint32_t rh[4], ih[4], rl[4], il[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        rh[e] = tf32_rna_bits(re[e]);
                        ih[e] = tf32_rna_bits(im[e]);
                        rl[e] = tf32_rna_bits(__float_as_uint(__uint_as_float(re[e]) - __uint_as_float(rh[e])));
                        il[e] = tf32_rna_bits(__float_as_uint(__uint_as_float(im[e]) - __uint_as_float(ih[e])));
                    }
                    *reinterpret_cast<uint4*>(stg + ihi[k][0]) = make_uint4(rh[0], rh[1], rh[2], rh[3]);
                    *reinterpret_cast<uint4*>(stg + ihi[k][1]) = make_uint4(ih[0], ih[1], ih[2], ih[3]);
                    *reinterpret_cast<uint4*>(stg + ilo[k][0]) = make_uint4(rl[0], rl[1], rl[2], rl[3]);
                    *reinterpret_cast<uint4*>(stg + ilo[k][1]) = make_uint4(il[0], il[1], il[2], il[3]);
                }
            }
            fence_proxy_async();  // the stores, seen by the tensor cores' async proxy
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(FULL + s));
        }
        cp_async_wait_all();
    } else if (warp == WS_MMA_WARP) {
        // ---- MMA issuer
        bool issued_any = false;
        if (lane == 0) {
#pragma unroll 1
            for (int t = 0; t < nt; ++t) {
                const int s = t % WS_STAGES, b = t % WS_NACC;
                if (!mbar_wait(bar(ACCE + b), (uint32_t)(((t / WS_NACC) & 1) ^ 1), abort_flag)) {
                    ok = false;
                    break;
                }
                if (!mbar_wait(bar(FULL + s), (uint32_t)((t / WS_STAGES) & 1), abort_flag)) {
                    ok = false;
                    break;
                }
                fence_after();
                const uint32_t st = base + (uint32_t)s * g.stage_bytes;
                const uint32_t dm = tmem + (uint32_t)(b * BN);
                const uint32_t dc = tmem + (uint32_t)(WS_NACC * BN);
#pragma unroll
                for (int kk = 0; kk < BK / 8; ++kk) {
                    const uint64_t ahi = sw128_desc(st + kk * 32);
                    const uint64_t alo = sw128_desc(st + A_PART + kk * 32);
                    const uint64_t bhi = sw128_desc(st + 2 * A_PART + kk * 32);
                    const uint64_t blo = sw128_desc(st + 2 * A_PART + b_part + kk * 32);
                    mma_tf32_n(dm, ahi, bhi, idesc, kk > 0 ? 1u : 0u);
                    mma_tf32_n(dc, alo, bhi, idesc, (t > 0 || kk > 0) ? 1u : 0u);
                    mma_tf32_n(dc, ahi, blo, idesc, 1u);
                }
                issued_any = true;
                mma_commit(bar(EMPTY + s));
                mma_commit(bar(ACCF + b));
            }
            // every MMA issued has completed before the teardown frees tensor memory
            if (issued_any) {
                mma_commit(bar(DRAIN));
                mbar_drain(bar(DRAIN), 0);
            }
        }
        __syncwarp();
    } else {
        // ---- drain warps
        const int q = warp & 3;
        // columns of this warp: its share of the groups of 8
        constexpr int PARTS = DRAINS / 4, WS_MAX_DC = (PARTS == 2 ? WS_MAX_NB8 : WS_MAX_NB) / PARTS;
        const int h = (warp - WS_DRAIN_WARP0) >> 2;
        const int col0 = nb / 8 * h / PARTS * 8, dc = nb / 8 * (h + 1) / PARTS * 8 - col0;
        const uint32_t lane_base = tmem + ((uint32_t)(32 * q) << 16);
        double acc[WS_MAX_DC];
#pragma unroll
        for (int i = 0; i < WS_MAX_DC; ++i) acc[i] = 0.0;
        const auto add_cols = [&](uint32_t col) {
#pragma unroll
            for (int j = 0; j < WS_MAX_DC / 8; ++j) {
                if (8 * j < dc) {
                    float v[8];
                    tmem_ld8(lane_base + col + (uint32_t)(col0 + 8 * j), v);
#pragma unroll
                    for (int i = 0; i < 8; ++i) acc[8 * j + i] += (double)v[i];
                }
            }
        };
        // two k-tiles' main products (buffers at columns c0 and c1), loaded under one wait.  PAIRS: their FP32
        // sum, rounded to nearest once (unbiased, 2^-24 of the pair against the TF32x3 parts' 2^-22 of each
        // product), goes into the FP64 sums -- half the conversions of one by one
        const auto add_pair = [&](uint32_t c0, uint32_t c1) {
#pragma unroll
            for (int j = 0; j < WS_MAX_DC / 8; ++j) {
                if (8 * j < dc) {
                    uint32_t r[16];
                    tmem_ld8_issue(lane_base + c0 + (uint32_t)(col0 + 8 * j), r);
                    tmem_ld8_issue(lane_base + c1 + (uint32_t)(col0 + 8 * j), r + 8);
                    tmem_wait_ld16(r);
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (PAIRS) {
                            acc[8 * j + i] += (double)(__uint_as_float(r[i]) + __uint_as_float(r[8 + i]));
                        } else {
                            acc[8 * j + i] += (double)__uint_as_float(r[i]);
                            acc[8 * j + i] += (double)__uint_as_float(r[8 + i]);
                        }
                }
            }
        };
#pragma unroll 1
        for (int t = 0; t < nt; t += 2) {
            const bool pair = t + 1 < nt;
            const int b0 = t % WS_NACC, b1 = (t + 1) % WS_NACC;
            bool got = mbar_wait(bar(ACCF + b0), (uint32_t)((t / WS_NACC) & 1), abort_flag);
            if (got && pair) got = mbar_wait(bar(ACCF + b1), (uint32_t)(((t + 1) / WS_NACC) & 1), abort_flag);
            if (!__all_sync(0xffffffffu, got)) {
                ok = false;
                break;
            }
            fence_after();
            if (pair)
                add_pair((uint32_t)(b0 * BN), (uint32_t)(b1 * BN));
            else
                add_cols((uint32_t)(b0 * BN));
            fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(bar(ACCE + b0));
                if (pair) mbar_arrive(bar(ACCE + b1));
            }
        }
        if (ok) {
            // the correction accumulator is complete with the last k-tile's commit
            fence_after();
            add_cols((uint32_t)(WS_NACC * BN));
            const int R = 32 * q + lane;
            const int l = R >> 1, pa = R & 1;
            if (l < nA) {
                double* row = g.out4 + ((long long)(la0 + l) * g.tiles.ldr + rb0) * 4;
#pragma unroll
                for (int j = 0; j < WS_MAX_DC; ++j) {
                    const int Cg = col0 + j;
                    const int r = Cg >> 1, pc = Cg & 1;
                    if (j < dc && r < nB) {
                        const int qi = (pa == pc) ? pa : 2 + pa;  // ac, bd, ad, bc
                        atomicAdd(row + 4 * r + qi, acc[j]);
                    }
                }
            }
        }
    }

    fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag)
        *reinterpret_cast<volatile int*>(g.err) = 1;
    if (warp == 0) {
        __syncwarp();
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

}  // namespace tc
}  // namespace clk
