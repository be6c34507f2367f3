// Quadrant plane passes of the sub-lattice forms for planes of two different lengths: the passes of
// plane_w.cuh with the y transform chosen at run time among the compiled lengths.
//
// A kernel per pair of lengths would be 22 x 22 of them each way.  The kernels are compiled per x length
// and call one function per y length (not inlined, so a translation unit holds each once); the call, and
// a row pitch known only at run time, cost little beside the stages themselves.
//
// Measured on a B200 against the separate x and y passes (forward and inverse together, 36 densities): 24 x
// 32 x 20 cells 0.184 -> 0.132 ms, 40 x 32 x 24 0.340 -> 0.212, 64 x 48 x 16 0.520 -> 0.311, 12 x 64 x 30
// 0.266 -> 0.203; 54 x 72 x 80 grid, two classes, 0.129 -> 0.112.
#pragma once

#include "plane_w.cuh"

namespace clk {
namespace pw {

// Items e = x + Q k of a column stage, x < Q, dealt to the block's threads: (x, k) of the first one and
// of the next.
struct ColumnItem {
    int x, k;
    __device__ ColumnItem(int Q) : x((int)threadIdx.x % Q), k((int)threadIdx.x / Q) {}
    __device__ void next(int Q, int dx, int dk) {
        x += dx;
        k += dk;
        if (x >= Q) {
            x -= Q;
            ++k;
        }
    }
};

// y transform of the Q columns of I (rows of `pitch` values), inputs in rows [0, N / 2): row R2 q + s holds
// frequency q + R1 s.  Ends with a barrier.
template <int H, int R2, typename T>
__device__ __noinline__ void y_forward(cx<T>* I, int pitch, int Q, const cx<T>* tw) {
    constexpr int R1 = 2 * H;
    const int dx = (int)blockDim.x % Q, dk = (int)blockDim.x / Q;
#pragma unroll 1
    for (ColumnItem i(Q); i.k < R2; i.next(Q, dx, dk)) {
        cx<T>* c = I + i.k * pitch + i.x;
        const int step = R2 * pitch;
        cx<T> v[H], ev[H], od[H];
#pragma unroll
        for (int j = 0; j < H; ++j) v[j] = c[j * step];
        dft_zero_padded<H>(v, ev, od);
#pragma unroll
        for (int k = 0; k < H; ++k) {
            c[(2 * k) * step] = ev[k];
            c[(2 * k + 1) * step] = od[k];
        }
    }
    __syncthreads();
#pragma unroll 1
    for (ColumnItem i(Q); i.k < R1; i.next(Q, dx, dk)) {
        cx<T>* c = I + (R2 * i.k) * pitch + i.x;
        cx<T> u[R2];
#pragma unroll
        for (int t = 0; t < R2; ++t) u[t] = t == 0 ? c[0] : cmul(c[t * pitch], tw[t * R1 + i.k]);
        dft<R2, -1, true>(u);
#pragma unroll
        for (int s = 0; s < R2; ++s) c[s * pitch] = u[s];
    }
    __syncthreads();
}

// Inverse y transform of the Q columns, rows in natural frequency order; outputs y < N / 2 to the atoms.
template <int H, int R2, typename T>
__device__ __noinline__ void y_inverse(cx<T>* I, int pitch, int Q, const cx<T>* tw, const Occupancy& occ,
                                       cx<T>* op) {
    constexpr int R1 = 2 * H;
    const int dx = (int)blockDim.x % Q, dk = (int)blockDim.x / Q;
#pragma unroll 1
    for (ColumnItem i(Q); i.k < R1; i.next(Q, dx, dk)) {
        cx<T>* c = I + i.k * pitch + i.x;
        const int step = R1 * pitch;
        cx<T> u[R2];
#pragma unroll
        for (int s = 0; s < R2; ++s) u[s] = c[s * step];
        dft<R2, +1, true>(u);
#pragma unroll
        for (int t = 0; t < R2; ++t) c[t * step] = t == 0 ? u[0] : cmulc(u[t], tw[t * R1 + i.k]);
    }
    __syncthreads();
#pragma unroll 1
    for (ColumnItem i(Q); i.k < R2; i.next(Q, dx, dk)) {
        const cx<T>* c = I + (R1 * i.k) * pitch + i.x;
        cx<T> ev[H], od[H];
#pragma unroll
        for (int k = 0; k < H; ++k) {
            ev[k] = c[(2 * k) * pitch];
            od[k] = c[(2 * k + 1) * pitch];
        }
        idft_first_half<H>(ev, od);
        int a[H];
#pragma unroll
        for (int n = 0; n < H; ++n) a[n] = atom_at(occ, i.x, i.k + R2 * n, Q);
#pragma unroll
        for (int n = 0; n < H; ++n)
            if (a[n] >= 0) op[a[n]] = ev[n];
    }
}

// R2 of a y length's split.
__device__ __forceinline__ int plane_r2(int n) {
    int r2 = 1;
    with_plane_w_device(n, [&](auto tag) { r2 = decltype(tag)::r2; });
    return r2;
}

template <typename T, int H, int R2, bool FWD>
struct PlaneXY {
    using L = PlaneW<T, H, R2, FWD>;
    // the FP64 inverse keeps its next rows in registers across the call: 168 a thread, 255 for 256 threads
    // (48 x 40 x 24 cells: 0.363 ms, 0.459 when held to 128)
    static constexpr int THREADS = L::THREADS, MIN = sizeof(T) == 8 && !FWD ? (384 / THREADS) : L::MOST;
    static size_t smem(int ny) {
        return sizeof(cx<T>) * ((size_t)ny * L::PQ + (size_t)L::RB * L::SP + L::N + ny) + 3 * (ny / 2) * sizeof(unsigned);
    }
    static int resident(int ny) {
        const int fit = (int)(228 * 1024 / (smem(ny) + 1024));
        return fit < 1 ? 1 : fit < MIN ? fit : MIN;
    }
};

template <typename T, int H, int R2>
__global__ void __launch_bounds__(PlaneXY<T, H, R2, true>::THREADS, PlaneXY<T, H, R2, true>::MIN)
    k_pfwd_xy(const cx<T>* __restrict__ rho, long long rho_stride, const int* __restrict__ row_ptr,
              const unsigned long long* __restrict__ row_mask, cx<T>* __restrict__ out, long long out_stride,
              const cx<T>* __restrict__ twx_g, const cx<T>* __restrict__ twy_g, int ny, int np) {
    using L = PlaneW<T, H, R2, true>;
    constexpr int R1 = L::R1, N = L::N, Q = L::Q, PQ = L::PQ, TP = L::TP, SP = L::SP, RB = L::RB, THREADS = L::THREADS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int qy = ny / 2, ry2 = plane_r2(ny), ry1 = ny / ry2;
    cx<T>* I = reinterpret_cast<cx<T>*>(smem_raw);
    cx<T>* S = I + ny * PQ;
    cx<T>* tw = S + RB * SP;
    cx<T>* twy = tw + N;
    const int tid = threadIdx.x, z = blockIdx.x;
    for (int i = tid; i < N; i += THREADS) tw[i] = twx_g[(i / R1) * (i % R1)];
    for (int i = tid; i < ny; i += THREADS) twy[i] = twy_g[(i / ry1) * (i % ry1)];
    const int a0 = row_ptr[z * ny], a1 = row_ptr[z * ny + ny];
    const Occupancy occ = plane_occupancy(reinterpret_cast<unsigned*>(twy + ny), row_ptr, row_mask, z, a0, a1, Q, qy, ny);
    const int per = (np + gridDim.y - 1) / gridDim.y;
    const int p_begin = blockIdx.y * per, p_end = min(np, p_begin + per);
    constexpr int PER = 16 / (int)sizeof(cx<T>);  // values a 16-byte copy
    const bool whole = occ.full && Q % PER == 0 && PQ % PER == 0 && rho_stride % PER == 0 &&
                       reinterpret_cast<uintptr_t>(rho + a0) % 16 == 0;
    const auto copy_in = [&](int p) {
        const cx<T>* src = rho + (long long)p * rho_stride + a0;
        if (whole) {
            for (int e = tid; e < Q * qy / PER; e += THREADS) {
                const int y = e / (Q / PER), x = PER * (e % (Q / PER));
                pd_cp_async16(I + y * PQ + x, src + PER * e);
            }
        } else {
            for (int e = tid; e < Q * qy; e += THREADS) {
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
        with_plane_w_device(ny, [&](auto tag) { y_forward<decltype(tag)::r1, decltype(tag)::r2>(I, PQ, Q, twy); });
        cx<T>* o = out + (long long)p * out_stride + (long long)z * N * ny;
        bool copied = false;
#pragma unroll 1
        for (int r0 = 0; r0 < ny; r0 += RB) {
            const int rows = min(RB, ny - r0);
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
            if (!copied && r0 + RB >= qy) {  // rows [0, qy) of I have been read
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
                cx<T>* orow = o + (r / ry2 + ry1 * (r % ry2)) * N + q;
#pragma unroll
                for (int s = 0; s < R2; ++s) orow[R1 * s] = u[s];
            }
            if (r0 + RB < ny) __syncthreads();  // the scratch is refilled
        }
    }
}

template <typename T, int H, int R2>
__global__ void __launch_bounds__(PlaneXY<T, H, R2, false>::THREADS, PlaneXY<T, H, R2, false>::MIN)
    k_pinv_xy(const cx<T>* __restrict__ buf, long long stride, const cx<T>* __restrict__ twx_g,
              const cx<T>* __restrict__ twy_g, const int* __restrict__ row_ptr, const unsigned long long* __restrict__ row_mask,
              cx<T>* __restrict__ out, long long o_stride, int ny, int np) {
    using L = PlaneW<T, H, R2, false>;
    constexpr int R1 = L::R1, N = L::N, Q = L::Q, PQ = L::PQ, TP = L::TP, SP = L::SP, RB = L::RB, THREADS = L::THREADS;
    constexpr int IX = (RB * R1 + THREADS - 1) / THREADS;  // first-stage items of a thread
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int qy = ny / 2, ry1 = ny / plane_r2(ny);
    cx<T>* I = reinterpret_cast<cx<T>*>(smem_raw);
    cx<T>* S = I + ny * PQ;
    cx<T>* tw = S + RB * SP;
    cx<T>* twy = tw + N;
    const int tid = threadIdx.x, z = blockIdx.x;
    for (int i = tid; i < N; i += THREADS) tw[i] = twx_g[(i / R1) * (i % R1)];
    for (int i = tid; i < ny; i += THREADS) twy[i] = twy_g[(i / ry1) * (i % ry1)];
    const int a0 = row_ptr[z * ny], a1 = row_ptr[z * ny + ny];
    const Occupancy occ = plane_occupancy(reinterpret_cast<unsigned*>(twy + ny), row_ptr, row_mask, z, a0, a1, Q, qy, ny);
    const int per = (np + gridDim.y - 1) / gridDim.y;
    const int p_begin = blockIdx.y * per, p_end = min(np, p_begin + per);
    cx<T> v[IX][R2];
    const auto load = [&](int p, int r0) {  // rows r0.. of density p
        const cx<T>* src = buf + (long long)p * stride + (long long)z * N * ny;
#pragma unroll
        for (int a = 0; a < IX; ++a) {
            const int e = tid + a * THREADS, q = e % R1, r = r0 + e / R1;
#pragma unroll
            for (int s = 0; s < R2; ++s) v[a][s] = (e < RB * R1 && r < ny) ? src[r * N + q + R1 * s] : mk(T(0), T(0));
        }
    };
    if (p_begin < p_end) load(p_begin, 0);
    for (int p = p_begin; p < p_end; ++p) {
#pragma unroll 1
        for (int r0 = 0; r0 < ny; r0 += RB) {
            const int rows = min(RB, ny - r0);
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
            if (r0 + RB < ny)
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
        cx<T>* op = out + (long long)p * o_stride + a0;
        with_plane_w_device(ny, [&](auto tag) { y_inverse<decltype(tag)::r1, decltype(tag)::r2>(I, PQ, Q, twy, occ, op); });
        // I is rewritten only after the barrier that follows the next plane's first stage
    }
}

}  // namespace pw
}  // namespace clk
