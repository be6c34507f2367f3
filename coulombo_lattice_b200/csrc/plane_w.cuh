// Quadrant plane passes of the sub-lattice forms: the x and y transforms of a class plane in one
// kernel each way, for square planes of every length the class-mixing z pass serves (zmix_wht.cuh).
//
// A class plane of N x N points (N = 2n/m) holds atoms only in its [0, Q)^2 quadrant, Q = N / 2.  Forward,
// y is transformed first, on Q columns with half their inputs zero, then x; inverse, x first, keeping Q
// of its outputs, then y on Q columns, keeping Q.  N-point lines are 2 H R2 points, as in zmix_wht.cuh:
// R1 = 2 H points (half of them zero, or half the outputs kept) times R2.
//
// A block holds one plane's half-transformed quadrant in shared memory, I[N][PQ], and passes the x stage
// through a scratch S of RB rows.  What each density needs first is on its way while the one before it is
// finished: forward, the atoms go by cp.async into rows [0, Q) of I as soon as the x stage has read them;
// inverse, the next RB rows' (or the next plane's first) points are loaded into registers while the
// current ones are transformed.  The inverse writes its last stage's outputs straight to the atoms.
//
// Pitches, with W = 16 complex values (8 in FP64) a shared-memory wavefront: the x stage's lanes hold R2
// adjacent columns of consecutive rows, so PQ = R2 mod W puts W lanes on consecutive words; a scratch row
// holds item t's outputs at t TP, TP = ceil(W / R2) mod W and SP = 1 mod W, so that R2 x (W / R2) lanes hit
// distinct banks when written and consecutive lanes consecutive words when read.
//
// Bound: shared-memory wavefronts and latency at 16 warps an SM; HBM at 64-point planes.  Measured on a B200
// against the passes these replace (a whole plane in shared memory, one block an SM, and a quadrant forward
// pass, at 128 points; separate x and y passes at lengths without a plane pass): 36 densities of 128 x 128
// planes, 2.1M atoms, 0.889 -> 0.570 ms forward (5.3 TB/s) and 0.898 -> 0.746 inverse (4.1); 820 of 64 x
// 64, 1.94 -> 1.35 (6.4 TB/s) and 1.89 -> 1.57; 78 of 48 x 48, 0.159 -> 0.086 and 0.165 -> 0.087.
// In FP64: 78 densities of 48 x 48, 0.280 -> 0.138 ms and 0.281 -> 0.140; 36 of 128 x 128 (64 x 64 x 16
// cells), both ways, 1.08 -> 0.83.
#pragma once

#include "fft.cuh"
#include "kernels.cuh"
#include "zmix_wht.cuh"

namespace clk {
namespace pw {

// The least number from at_least up that is rest modulo w.
constexpr int up_to(int at_least, int rest, int w) { return at_least + ((rest - at_least) % w + w) % w; }

template <typename T, int H, int R2, bool FWD>
struct PlaneW {
    static constexpr int R1 = 2 * H, N = R1 * R2, Q = N / 2;
    static constexpr int W = 128 / (int)sizeof(cx<T>);  // values a shared-memory wavefront serves
    static constexpr int PQ = up_to(Q, R2 % W, W);
    static constexpr int TP = up_to(R1, (W + R2 - 1) / R2 % W, W);
    static constexpr int SP = up_to(R2 * TP, 1, W);
    // Threads, and x-stage rows at a time.  Measured in FP32 (a request's densities, ms): 128-point planes,
    // 256 threads with 32 rows 0.57 forward and 0.80 inverse, with 16 rows 0.60 and 0.74; 512 threads of 64
    // registers 0.63 and 0.76; 64-point planes, 128 threads with 32 rows 0.67 and 0.77, 256 threads 0.72
    // and 0.77, with all 64 rows 0.73 and 0.78; 48-point planes, all rows 0.082 and 0.081, half of them
    // 0.079 and 0.087.  FP64 planes are twice the size: half the rows, and 256 threads from 65 points on
    // (64-point planes, 36 densities, 128 threads 0.143 and 0.174, 256 threads 0.158 and 0.187; at 168
    // registers a thread, one block of 256 an SM, 0.158 and 0.297).
    static constexpr bool F32 = sizeof(T) == 4;
    static constexpr int THREADS = N > (F32 ? 96 : 64) ? 256 : 128;
    static constexpr int RB = F32 ? (N > 96 ? (FWD ? 32 : 16) : N > 48 ? (N + 1) / 2 : N)
                                  : (N > 96 ? 16 : N > 48 ? (N + 3) / 4 : (N + 1) / 2);
    static constexpr size_t smem = sizeof(cx<T>) * ((size_t)N * PQ + (size_t)RB * SP + N) + 3 * Q * sizeof(unsigned);
    static constexpr int kThreads = 512;  // resident at 128 registers
    static constexpr int fit = (int)(228 * 1024 / (smem + 1024));
    static constexpr int MOST = kThreads / THREADS < 1 ? 1 : kThreads / THREADS;
    static constexpr int MIN = fit < MOST ? (fit < 1 ? 1 : fit) : MOST;
};

// Which quadrant points of the plane hold atoms: 64 bits a row and the row's first atom.
struct Occupancy {
    unsigned* mask;  // [Q][2]
    unsigned* base;  // [Q], from the plane's first atom
    bool full;       // every quadrant point, in order
};
// (qx, qy): the quadrant; ny: rows of the plane; row_mask: the atoms of every row (k_row_masks).  Blocks that built
// the masks from their atoms' cells spent 5 us on it before the first copy: 96 x 96 planes with 92 x 92 atoms,
// one density 0.035 -> 0.026 ms forward and 0.038 -> 0.025 inverse, six 0.106 -> 0.080 and 0.112 -> 0.080.
__device__ __forceinline__ Occupancy plane_occupancy(unsigned* mem, const int* row_ptr,
                                                     const unsigned long long* row_mask, int z, int a0, int a1, int qx,
                                                     int qy, int ny) {
    Occupancy o{mem, mem + 2 * qy, a1 - a0 == qx * qy};
    if (!o.full)
        for (int y = threadIdx.x; y < qy; y += blockDim.x) {
            const unsigned long long m = row_mask[z * ny + y];
            o.base[y] = row_ptr[z * ny + y] - a0;
            o.mask[2 * y] = (unsigned)m;
            o.mask[2 * y + 1] = (unsigned)(m >> 32);
        }
    __syncthreads();
    return o;
}
// Index (from the plane's first atom) of the atom at (x, y) of a quadrant Q wide, or -1.
__device__ __forceinline__ int atom_at(const Occupancy& o, int x, int y, int Q) {
    if (o.full) return y * Q + x;
    const unsigned w0 = o.mask[2 * y], w = x < 32 ? w0 : o.mask[2 * y + 1];
    if (!((w >> (x & 31)) & 1u)) return -1;
    return (int)(o.base[y] + (x < 32 ? 0 : __popc(w0)) + __popc(w & ((1u << (x & 31)) - 1u)));
}

template <typename T, int H, int R2>
__global__ void __launch_bounds__(PlaneW<T, H, R2, true>::THREADS, PlaneW<T, H, R2, true>::MIN)
    k_pfwd(const cx<T>* __restrict__ rho, long long rho_stride, const int* __restrict__ row_ptr,
           const unsigned long long* __restrict__ row_mask, cx<T>* __restrict__ out, long long out_stride,
           const cx<T>* __restrict__ tw_g, int np) {
    using L = PlaneW<T, H, R2, true>;
    constexpr int R1 = L::R1, N = L::N, Q = L::Q, PQ = L::PQ, TP = L::TP, SP = L::SP, RB = L::RB, THREADS = L::THREADS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cx<T>* I = reinterpret_cast<cx<T>*>(smem_raw);
    cx<T>* S = I + N * PQ;
    cx<T>* tw = S + RB * SP;
    const int tid = threadIdx.x, z = blockIdx.x;
    for (int i = tid; i < N; i += THREADS) tw[i] = tw_g[(i / R1) * (i % R1)];  // [t][q]: W^(t q)
    const int a0 = row_ptr[z * N], a1 = row_ptr[z * N + N];
    const Occupancy occ = plane_occupancy(reinterpret_cast<unsigned*>(tw + N), row_ptr, row_mask, z, a0, a1, Q, Q, N);
    const int per = (np + gridDim.y - 1) / gridDim.y;
    const int p_begin = blockIdx.y * per, p_end = min(np, p_begin + per);
    constexpr int PER = 16 / (int)sizeof(cx<T>);  // values a 16-byte copy
    const bool whole = occ.full && Q % PER == 0 && PQ % PER == 0 && rho_stride % PER == 0 &&
                       reinterpret_cast<uintptr_t>(rho + a0) % 16 == 0;
    const auto copy_in = [&](int p) {
        const cx<T>* src = rho + (long long)p * rho_stride + a0;
        if (whole) {
            for (int e = tid; e < Q * Q / PER; e += THREADS) {
                const int y = e / (Q / PER), x = PER * (e % (Q / PER));
                pd_cp_async16(I + y * PQ + x, src + PER * e);
            }
        } else {
            for (int e = tid; e < Q * Q; e += THREADS) {
                const int y = e / Q, x = e % Q;
                const int i = atom_at(occ, x, y, Q);
                if (i >= 0)
                    cp_async<sizeof(cx<T>)>(I + y * PQ + x, src + i);
                else
                    I[y * PQ + x] = mk(T(0), T(0));
            }
        }
    };
    if (p_begin < p_end) copy_in(p_begin);
    for (int p = p_begin; p < p_end; ++p) {
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();
        // y, first stage: columns x < Q, inputs y < Q; item t's output q to row t + R2 q
#pragma unroll 1
        for (int e = tid; e < Q * R2; e += THREADS) {
            const int x = e % Q, t = e / Q;
            cx<T>* c = I + t * PQ + x;
            cx<T> v[H], ev[H], od[H];
#pragma unroll
            for (int j = 0; j < H; ++j) v[j] = c[(R2 * j) * PQ];
            dft_zero_padded<H>(v, ev, od);
#pragma unroll
            for (int k = 0; k < H; ++k) {
                c[(R2 * (2 * k)) * PQ] = ev[k];
                c[(R2 * (2 * k + 1)) * PQ] = od[k];
            }
        }
        __syncthreads();
        // y, second stage: row R2 q + s then holds frequency ky = q + R1 s
#pragma unroll 2
        for (int e = tid; e < Q * R1; e += THREADS) {
            const int x = e % Q, q = e / Q;
            cx<T>* c = I + (R2 * q) * PQ + x;
            cx<T> u[R2];
#pragma unroll
            for (int t = 0; t < R2; ++t) u[t] = t == 0 ? c[0] : cmul(c[t * PQ], tw[t * R1 + q]);
            dft<R2, -1, true>(u);
#pragma unroll
            for (int s = 0; s < R2; ++s) c[s * PQ] = u[s];
        }
        __syncthreads();
        cx<T>* o = out + (long long)p * out_stride + (long long)z * N * N;
        bool copied = false;
#pragma unroll 1
        for (int r0 = 0; r0 < N; r0 += RB) {
            const int rows = min(RB, N - r0);
            // x, first stage, into the scratch
#pragma unroll 1
            for (int e = tid; e < rows * R2; e += THREADS) {
                const int t = e % R2, rr = e / R2;
                const cx<T>* c = I + (r0 + rr) * PQ + t;
                cx<T> v[H], ev[H], od[H];
#pragma unroll
                for (int j = 0; j < H; ++j) v[j] = c[R2 * j];
                dft_zero_padded<H>(v, ev, od);
                cx<T>* d = S + rr * SP + t * TP;
#pragma unroll
                for (int k = 0; k < H; ++k) {
                    d[2 * k] = ev[k];
                    d[2 * k + 1] = od[k];
                }
            }
            __syncthreads();
            if (!copied && r0 + RB >= Q) {  // rows [0, Q) of I have been read
                copied = true;
                if (p + 1 < p_end) copy_in(p + 1);
            }
            // x, second stage, to HBM
#pragma unroll 2
            for (int e = tid; e < rows * R1; e += THREADS) {
                const int q = e % R1, rr = e / R1, r = r0 + rr;
                const cx<T>* d = S + rr * SP + q;
                cx<T> u[R2];
#pragma unroll
                for (int t = 0; t < R2; ++t) u[t] = t == 0 ? d[0] : cmul(d[t * TP], tw[t * R1 + q]);
                dft<R2, -1, true>(u);
                cx<T>* orow = o + (r / R2 + R1 * (r % R2)) * N + q;
#pragma unroll
                for (int s = 0; s < R2; ++s) orow[R1 * s] = u[s];
            }
            if (r0 + RB < N) __syncthreads();  // the scratch is refilled
        }
    }
}

template <typename T, int H, int R2>
__global__ void __launch_bounds__(PlaneW<T, H, R2, false>::THREADS, PlaneW<T, H, R2, false>::MIN)
    k_pinv(const cx<T>* __restrict__ buf, long long stride, const cx<T>* __restrict__ tw_g,
           const int* __restrict__ row_ptr, const unsigned long long* __restrict__ row_mask, cx<T>* __restrict__ out,
           long long o_stride, int np) {
    using L = PlaneW<T, H, R2, false>;
    constexpr int R1 = L::R1, N = L::N, Q = L::Q, PQ = L::PQ, TP = L::TP, SP = L::SP, RB = L::RB, THREADS = L::THREADS;
    constexpr int IX = (RB * R1 + THREADS - 1) / THREADS;  // first-stage items of a thread
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cx<T>* I = reinterpret_cast<cx<T>*>(smem_raw);
    cx<T>* S = I + N * PQ;
    cx<T>* tw = S + RB * SP;
    const int tid = threadIdx.x, z = blockIdx.x;
    for (int i = tid; i < N; i += THREADS) tw[i] = tw_g[(i / R1) * (i % R1)];  // [t][q]: W^(t q)
    const int a0 = row_ptr[z * N], a1 = row_ptr[z * N + N];
    const Occupancy occ = plane_occupancy(reinterpret_cast<unsigned*>(tw + N), row_ptr, row_mask, z, a0, a1, Q, Q, N);
    const int per = (np + gridDim.y - 1) / gridDim.y;
    const int p_begin = blockIdx.y * per, p_end = min(np, p_begin + per);
    cx<T> v[IX][R2];
    const auto load = [&](int p, int r0) {  // rows r0.. of density p
        const cx<T>* src = buf + (long long)p * stride + (long long)z * N * N;
#pragma unroll
        for (int a = 0; a < IX; ++a) {
            const int e = tid + a * THREADS, q = e % R1, r = r0 + e / R1;
#pragma unroll
            for (int s = 0; s < R2; ++s) v[a][s] = (e < RB * R1 && r < N) ? src[r * N + q + R1 * s] : mk(T(0), T(0));
        }
    };
    if (p_begin < p_end) load(p_begin, 0);
    for (int p = p_begin; p < p_end; ++p) {
#pragma unroll 1
        for (int r0 = 0; r0 < N; r0 += RB) {
            const int rows = min(RB, N - r0);
            // x, first stage, from registers into the scratch
#pragma unroll
            for (int a = 0; a < IX; ++a) {
                const int e = tid + a * THREADS, q = e % R1, rr = e / R1;
                if (rr < rows) {
                    dft<R2, +1, true>(v[a]);
                    cx<T>* d = S + rr * SP + q;
#pragma unroll
                    for (int t = 0; t < R2; ++t) d[t * TP] = t == 0 ? v[a][0] : cmulc(v[a][t], tw[t * R1 + q]);
                }
            }
            __syncthreads();
            if (r0 + RB < N)
                load(p, r0 + RB);
            else if (p + 1 < p_end)
                load(p + 1, 0);
            // x, second stage: outputs x = t + R2 n < Q
#pragma unroll 1
            for (int e = tid; e < rows * R2; e += THREADS) {
                const int t = e % R2, rr = e / R2;
                const cx<T>* d = S + rr * SP + t * TP;
                cx<T> ev[H], od[H];
#pragma unroll
                for (int k = 0; k < H; ++k) {
                    ev[k] = d[2 * k];
                    od[k] = d[2 * k + 1];
                }
                idft_first_half<H>(ev, od);
                cx<T>* c = I + (r0 + rr) * PQ + t;
#pragma unroll
                for (int n = 0; n < H; ++n) c[R2 * n] = ev[n];
            }
            __syncthreads();
        }
        // y, first stage: rows ky = q + R1 s of a column, in place
#pragma unroll 2
        for (int e = tid; e < Q * R1; e += THREADS) {
            const int x = e % Q, q = e / Q;
            cx<T>* c = I + q * PQ + x;
            cx<T> u[R2];
#pragma unroll
            for (int s = 0; s < R2; ++s) u[s] = c[(R1 * s) * PQ];
            dft<R2, +1, true>(u);
#pragma unroll
            for (int t = 0; t < R2; ++t) c[(R1 * t) * PQ] = t == 0 ? u[0] : cmulc(u[t], tw[t * R1 + q]);
        }
        __syncthreads();
        // y, second stage: outputs y = t + R2 n < Q, to the atoms
        cx<T>* op = out + (long long)p * o_stride + a0;
#pragma unroll 1
        for (int e = tid; e < Q * R2; e += THREADS) {
            const int x = e % Q, t = e / Q;
            const cx<T>* c = I + (R1 * t) * PQ + x;
            cx<T> ev[H], od[H];
#pragma unroll
            for (int k = 0; k < H; ++k) {
                ev[k] = c[(2 * k) * PQ];
                od[k] = c[(2 * k + 1) * PQ];
            }
            idft_first_half<H>(ev, od);
            int i[H];
#pragma unroll
            for (int n = 0; n < H; ++n) i[n] = atom_at(occ, x, t + R2 * n, Q);
#pragma unroll
            for (int n = 0; n < H; ++n)
                if (i[n] >= 0) op[i[n]] = ev[n];
        }
        // I is rewritten only after the barrier that follows the next plane's first stage
    }
}

// The compiled splits N = 2 H R2 of the plane lengths; f is called with (H, R2) as SplitTag<H, R2>.
#define CLK_PW_LENGTHS(X)                                                                              \
    X(12, 3, 2) X(16, 4, 2) X(18, 3, 3) X(20, 5, 2) X(24, 4, 3) X(30, 5, 3) \
    X(32, 4, 4) X(36, 6, 3) X(40, 5, 4) X(48, 8, 3) X(50, 5, 5) X(54, 9, 3) \
    X(60, 6, 5) X(64, 8, 4) X(72, 9, 4) X(80, 8, 5) X(90, 9, 5) X(96, 8, 6) \
    X(100, 10, 5) X(108, 9, 6) X(120, 10, 6) X(128, 8, 8)
#define CLK_PW_CASE(N, A, B) \
    case N:                  \
        f(SplitTag<A, B>{}); \
        return true;
template <typename F>
bool with_plane_w(int n, F&& f) {
    switch (n) {
        CLK_PW_LENGTHS(CLK_PW_CASE)
        default: return false;
    }
}
template <typename F>
__device__ __forceinline__ bool with_plane_w_device(int n, F&& f) {
    switch (n) {
        CLK_PW_LENGTHS(CLK_PW_CASE)
        default: return false;
    }
}

}  // namespace pw
}  // namespace clk
