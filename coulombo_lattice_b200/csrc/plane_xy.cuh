// Quadrant plane passes of the FP32 sub-lattice forms for planes of two different lengths: the passes of
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
template <int H, int R2>
__device__ __noinline__ void y_forward(cx<float>* I, int pitch, int Q, const cx<float>* tw) {
    constexpr int R1 = 2 * H;
    const int dx = (int)blockDim.x % Q, dk = (int)blockDim.x / Q;
#pragma unroll 1
    for (ColumnItem i(Q); i.k < R2; i.next(Q, dx, dk)) {
        cx<float>* c = I + i.k * pitch + i.x;
        const int step = R2 * pitch;
        cx<float> v[H], ev[H], od[H];
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
        cx<float>* c = I + (R2 * i.k) * pitch + i.x;
        cx<float> u[R2];
#pragma unroll
        for (int t = 0; t < R2; ++t) u[t] = t == 0 ? c[0] : cmul(c[t * pitch], tw[t * R1 + i.k]);
        dft<R2, -1>(u);
#pragma unroll
        for (int s = 0; s < R2; ++s) c[s * pitch] = u[s];
    }
    __syncthreads();
}

// Inverse y transform of the Q columns, rows in natural frequency order; outputs y < N / 2 to the atoms.
template <int H, int R2>
__device__ __noinline__ void y_inverse(cx<float>* I, int pitch, int Q, const cx<float>* tw, const Occupancy& occ,
                                       cx<float>* op) {
    constexpr int R1 = 2 * H;
    const int dx = (int)blockDim.x % Q, dk = (int)blockDim.x / Q;
#pragma unroll 1
    for (ColumnItem i(Q); i.k < R1; i.next(Q, dx, dk)) {
        cx<float>* c = I + i.k * pitch + i.x;
        const int step = R1 * pitch;
        cx<float> u[R2];
#pragma unroll
        for (int s = 0; s < R2; ++s) u[s] = c[s * step];
        dft<R2, +1>(u);
#pragma unroll
        for (int t = 0; t < R2; ++t) c[t * step] = t == 0 ? u[0] : cmulc(u[t], tw[t * R1 + i.k]);
    }
    __syncthreads();
#pragma unroll 1
    for (ColumnItem i(Q); i.k < R2; i.next(Q, dx, dk)) {
        const cx<float>* c = I + (R1 * i.k) * pitch + i.x;
        cx<float> ev[H], od[H];
#pragma unroll
        for (int k = 0; k < H; ++k) {
            ev[k] = c[(2 * k) * pitch];
            od[k] = c[(2 * k + 1) * pitch];
        }
        idft_first_half<H>(ev, od);
#pragma unroll
        for (int n = 0; n < H; ++n) {
            const int a = atom_at(occ, i.x, i.k + R2 * n, Q);
            if (a >= 0) op[a] = ev[n];
        }
    }
}

// R2 of a y length's split.
__device__ __forceinline__ int plane_r2(int n) {
    int r2 = 1;
    with_plane_w_device(n, [&](auto tag) { r2 = decltype(tag)::r2; });
    return r2;
}

template <int H, int R2, bool FWD>
struct PlaneXY {
    using L = PlaneW<H, R2, FWD>;
    static constexpr int THREADS = L::THREADS, MIN = 512 / THREADS;  // <= 128 registers
    static size_t smem(int ny) {
        return sizeof(cx<float>) * ((size_t)ny * L::PQ + (size_t)L::RB * L::SP + L::N + ny) + 3 * (ny / 2) * sizeof(unsigned);
    }
    static int resident(int ny) {
        const int fit = (int)(228 * 1024 / (smem(ny) + 1024));
        return fit < 1 ? 1 : fit < MIN ? fit : MIN;
    }
};

template <int H, int R2>
__global__ void __launch_bounds__(PlaneXY<H, R2, true>::THREADS, PlaneXY<H, R2, true>::MIN)
    k_pfwd_xy(const cx<float>* __restrict__ rho, long long rho_stride, const int* __restrict__ row_ptr,
              const int* __restrict__ cell, cx<float>* __restrict__ out, long long out_stride,
              const cx<float>* __restrict__ twx_g, const cx<float>* __restrict__ twy_g, int ny, int np) {
    using L = PlaneW<H, R2, true>;
    constexpr int R1 = L::R1, N = L::N, Q = L::Q, PQ = L::PQ, TP = L::TP, SP = L::SP, RB = L::RB, THREADS = L::THREADS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int qy = ny / 2, ry2 = plane_r2(ny), ry1 = ny / ry2;
    cx<float>* I = reinterpret_cast<cx<float>*>(smem_raw);
    cx<float>* S = I + ny * PQ;
    cx<float>* tw = S + RB * SP;
    cx<float>* twy = tw + N;
    const int tid = threadIdx.x, z = blockIdx.x;
    for (int i = tid; i < N; i += THREADS) tw[i] = twx_g[(i / R1) * (i % R1)];
    for (int i = tid; i < ny; i += THREADS) twy[i] = twy_g[(i / ry1) * (i % ry1)];
    const int a0 = row_ptr[z * ny], a1 = row_ptr[z * ny + ny];
    const Occupancy occ = plane_occupancy(reinterpret_cast<unsigned*>(twy + ny), row_ptr, cell, z, a0, a1, Q, qy, N, ny);
    const int per = (np + gridDim.y - 1) / gridDim.y;
    const int p_begin = blockIdx.y * per, p_end = min(np, p_begin + per);
    const bool pairs = occ.full && Q % 2 == 0 && PQ % 2 == 0 && rho_stride % 2 == 0 &&
                       reinterpret_cast<uintptr_t>(rho + a0) % 16 == 0;
    const auto copy_in = [&](int p) {
        const cx<float>* src = rho + (long long)p * rho_stride + a0;
        if (pairs) {
            for (int e = tid; e < Q * qy / 2; e += THREADS) {
                const int y = e / (Q / 2), x = 2 * (e % (Q / 2));
                pd_cp_async16(I + y * PQ + x, src + 2 * e);
            }
        } else {
            for (int e = tid; e < Q * qy; e += THREADS) {
                const int y = e / Q, x = e % Q;
                const int i = atom_at(occ, x, y, Q);
                if (i >= 0)
                    cp_async<8>(I + y * PQ + x, src + i);
                else
                    I[y * PQ + x] = mk(0.f, 0.f);
            }
        }
    };
    if (p_begin < p_end) copy_in(p_begin);
    for (int p = p_begin; p < p_end; ++p) {
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();
        with_plane_w_device(ny, [&](auto tag) { y_forward<decltype(tag)::r1, decltype(tag)::r2>(I, PQ, Q, twy); });
        cx<float>* o = out + (long long)p * out_stride + (long long)z * N * ny;
        bool copied = false;
#pragma unroll 1
        for (int r0 = 0; r0 < ny; r0 += RB) {
            const int rows = min(RB, ny - r0);
            // x, first stage, into the scratch
#pragma unroll 1
            for (int e = tid; e < rows * R2; e += THREADS) {
                const int t = e % R2, rr = e / R2;
                const cx<float>* c = I + (r0 + rr) * PQ + t;
                cx<float> v[H], ev[H], od[H];
#pragma unroll
                for (int j = 0; j < H; ++j) v[j] = c[R2 * j];
                dft_zero_padded<H>(v, ev, od);
                cx<float>* d = S + rr * SP + t * TP;
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
                const cx<float>* d = S + rr * SP + q;
                cx<float> u[R2];
#pragma unroll
                for (int t = 0; t < R2; ++t) u[t] = t == 0 ? d[0] : cmul(d[t * TP], tw[t * R1 + q]);
                dft<R2, -1>(u);
                cx<float>* orow = o + (r / ry2 + ry1 * (r % ry2)) * N + q;
#pragma unroll
                for (int s = 0; s < R2; ++s) orow[R1 * s] = u[s];
            }
            if (r0 + RB < ny) __syncthreads();  // the scratch is refilled
        }
    }
}

template <int H, int R2>
__global__ void __launch_bounds__(PlaneXY<H, R2, false>::THREADS, PlaneXY<H, R2, false>::MIN)
    k_pinv_xy(const cx<float>* __restrict__ buf, long long stride, const cx<float>* __restrict__ twx_g,
              const cx<float>* __restrict__ twy_g, const int* __restrict__ row_ptr, const int* __restrict__ cell,
              cx<float>* __restrict__ out, long long o_stride, int ny, int np) {
    using L = PlaneW<H, R2, false>;
    constexpr int R1 = L::R1, N = L::N, Q = L::Q, PQ = L::PQ, TP = L::TP, SP = L::SP, RB = L::RB, THREADS = L::THREADS;
    constexpr int IX = (RB * R1 + THREADS - 1) / THREADS;  // first-stage items of a thread
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int qy = ny / 2, ry1 = ny / plane_r2(ny);
    cx<float>* I = reinterpret_cast<cx<float>*>(smem_raw);
    cx<float>* S = I + ny * PQ;
    cx<float>* tw = S + RB * SP;
    cx<float>* twy = tw + N;
    const int tid = threadIdx.x, z = blockIdx.x;
    for (int i = tid; i < N; i += THREADS) tw[i] = twx_g[(i / R1) * (i % R1)];
    for (int i = tid; i < ny; i += THREADS) twy[i] = twy_g[(i / ry1) * (i % ry1)];
    const int a0 = row_ptr[z * ny], a1 = row_ptr[z * ny + ny];
    const Occupancy occ = plane_occupancy(reinterpret_cast<unsigned*>(twy + ny), row_ptr, cell, z, a0, a1, Q, qy, N, ny);
    const int per = (np + gridDim.y - 1) / gridDim.y;
    const int p_begin = blockIdx.y * per, p_end = min(np, p_begin + per);
    cx<float> v[IX][R2];
    const auto load = [&](int p, int r0) {  // rows r0.. of density p
        const cx<float>* src = buf + (long long)p * stride + (long long)z * N * ny;
#pragma unroll
        for (int a = 0; a < IX; ++a) {
            const int e = tid + a * THREADS, q = e % R1, r = r0 + e / R1;
#pragma unroll
            for (int s = 0; s < R2; ++s) v[a][s] = (e < RB * R1 && r < ny) ? src[r * N + q + R1 * s] : mk(0.f, 0.f);
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
                    dft<R2, +1>(v[a]);
                    cx<float>* d = S + rr * SP + q;
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
                const cx<float>* d = S + rr * SP + t * TP;
                cx<float> ev[H], od[H];
#pragma unroll
                for (int k = 0; k < H; ++k) {
                    ev[k] = d[2 * k];
                    od[k] = d[2 * k + 1];
                }
                idft_first_half<H>(ev, od);
                cx<float>* c = I + (r0 + rr) * PQ + t;
#pragma unroll
                for (int n = 0; n < H; ++n) c[R2 * n] = ev[n];
            }
            __syncthreads();
        }
        cx<float>* op = out + (long long)p * o_stride + a0;
        with_plane_w_device(ny, [&](auto tag) { y_inverse<decltype(tag)::r1, decltype(tag)::r2>(I, PQ, Q, twy, occ, op); });
        // I is rewritten only after the barrier that follows the next plane's first stage
    }
}

}  // namespace pw
}  // namespace clk
